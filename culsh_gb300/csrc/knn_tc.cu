// Candidate distances and top-K on the 5th-generation tensor cores for
// queries whose candidate sets cover a large share of the dataset.
//
// Replaces, for such queries, the host collect/sort/unique of
// cuLSH_SearchTables.cu:321-364, the distance kernel of
// cuLSH_Kernels.cu:301-348 (launched by cuLSH_Querying.cu:284-343) and the
// top-K of cuLSH_Kernels.cu:356-456. Results are those of the exact FP32
// path: the same ids and bit-identical squared distances.
//
// Formulation. A query's candidates are marked in an N-bit membership row
// (k_cand_bitmap, candidates.cu). Tiles of 256 queries are multiplied with
// tiles of 128 points by tcgen05.mma: fp16 operands (each query row and the
// dataset scaled by a power of two), FP32 accumulators in TMEM, operands
// staged by TMA. The epilogue turns each accumulator into a key
//     t = |x|^2 + m q.x       (m = -2 / scales, per query)
// and three steps use the keys:
//  1. Sample pass: over every f-th point (f <= 16), the smallest key among
//     the candidates of each 32-point chunk. The K-th smallest of a query's
//     chunk minima belongs to K different candidates, so the upper end of its
//     error interval bounds the K-th distance from above (k_knn_limit).
//  2. Full pass: every candidate whose certified lower bound does not exceed
//     that limit is appended to the list of its (CTA, column slice, query)
//     in global memory. About f K candidates of a query survive, so the
//     epilogue is one comparison of a 32-column minimum almost everywhere.
//  3. Merge: the survivors of a query are cut at the K-th smallest key, the
//     exact FP32 lane-order distances of those K and of whatever their largest
//     distance does not exclude are computed, and (distance, id) sorted.
// A query whose survivors outgrow their lists is scanned exactly from its
// membership row (k_knn_scan_rows, candidates.cu).
//
// Error interval. With |q - qh| <= r_q, |x - xh| <= rho |x| + a for every row
// (measured when the rows are converted), g the accumulation, norm and
// lane-order terms (knn_gamma) and 2 |q| |x| <= |q|^2 + |x|^2 = S, the exact
// FP32 distance d differs from |x|^2 - 2 qh.xh + |q|^2 by at most kappa S + e,
// kappa = 1.01 (r_q / |q| + rho) + g and e = 2.02 |q| a. Since the bound is
// linear in |x|^2 it is folded into m:
//     d >= (1 - kappa) (|x|^2 + m_lo q.x + |q|^2) - e,  m_lo = -2 / (1 - kappa)
//     d <= (1 + kappa) (|x|^2 + m_up q.x + |q|^2) + e,  m_up = -2 / (1 + kappa)
// One fp16 product per element bounds d to about 2^-11 S; a split into two
// bf16 parts and three products (2^-13 S), with sorted lists kept in the
// epilogue, was the earlier form: 8.8 ms against 2.6 + 0.2 ms (both passes) at
// 9,973 queries, 1M x 100.
// Queries and datasets of small integers (|v| <= 256, D max|v|^2 < 2^24 and
// D (max v - min v)^2 < 2^24) have kappa = e = 0: every product, partial sum
// and norm is an integer below 2^24, the key plus |q|^2 is the exact distance
// and no row is read again.
//
// Work split: the (query tile, point tile) pairs are cut into gridDim.x
// contiguous ranges, one per persistent CTA, so that every CTA does the same
// number of tensor-core tiles. A CTA's range covers part of one or a few
// query tiles; for each it leaves one list per query and column slice (list
// set blockIdx.x + query tile, unique because the ranges are ordered), which
// the merge kernel combines.
//
// Roles: warp 0 issues TMA loads (point tiles into a ring of 64-column slabs,
// membership words and point norms into a second ring; the query tile once
// per query tile for D <= 128, otherwise slab by slab beside the points);
// warp 1 owns TMEM and issues tcgen05.mma (M = 128 twice, N = 128, K = 16
// per instruction) into two accumulator sets, so that the epilogue of one tile
// overlaps the products of the next; the other sixteen warps read TMEM with
// tcgen05.ld. Every mbarrier wait is bounded: on timeout the kernel raises
// kErrSpin, drains its copies and products, frees TMEM and returns; the host
// then reports the error.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "culsh_internal.cuh"
#include "topk_common.cuh"

namespace culsh {
namespace {

constexpr int KM = 128;                 // rows of one MMA (TMEM lanes)
constexpr int MQ = kKnnTileQ;           // queries per tile: two MMAs share a point tile
constexpr int BN = 128;                 // points per tile
constexpr int MH = MQ / KM;
constexpr int MW = MH;                  // MMA warps, one per half of the query tile
constexpr int NEPI = 16;                // epilogue warps
constexpr int kKnnThreads = 32 * (1 + MW + NEPI);
constexpr int NT = 32 * NEPI;           // one (query, accumulator set) each
constexpr int NCH = NT / MQ;            // warp groups: one per accumulator set, alternating tiles
constexpr int BW = BN / 32;             // membership words per query row and point tile
constexpr uint32_t kXSlab = (uint32_t)BN * 128;   // bytes of 64 columns of a point tile
constexpr uint32_t kQSlab = (uint32_t)MQ * 128;   // ... of a query tile
constexpr uint32_t kBmBytes = (uint32_t)MQ * BW * 4, kWBytes = (uint32_t)BN * 4;
constexpr uint32_t kEpStride = kBmBytes + kWBytes;
constexpr int kEpStages = 4;            // membership / norm ring stages
constexpr int kMaxOpStages = 6;         // operand ring stages
constexpr int kResidentD = 128;         // query tile kept in shared memory up to this dimension
static_assert(NCH * MQ == NT && NCH == 2, "one warp group, and one list per query, per accumulator set");
// Bounded waits: each poll suspends the thread in hardware for up to
// kKnnSuspendNs (it resumes as soon as the phase completes, and takes no issue
// slots meanwhile), at most kKnnPoll polls (a few seconds) in all.
constexpr uint32_t kKnnPoll = 1u << 18;
constexpr uint32_t kKnnSuspendNs = 16384;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(kKnnSuspendNs)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool bar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the phase of the given parity; on timeout raises the
// block's abort flag and kErrSpin.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err) {
    if (bar_test(bar, parity)) return true;
    for (uint32_t i = 0; i < kKnnPoll; ++i) {
        if (bar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicOr(err, kErrSpin);
    return false;
}
// Bounded wait that ignores the abort flag (draining at exit).
__device__ __forceinline__ void bar_drain(uint64_t* bar, uint32_t parity, int* err) {
    for (uint32_t i = 0; i < kKnnPoll; ++i)
        if (bar_try_wait(bar, parity)) return;
    atomicOr(err, kErrSpin);
}

__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(
            d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}
// One lane of the (converged) warp, the same on every call.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Starts loading the 16 accumulator columns [taddr, taddr + 16) of this
// thread's TMEM lane; r holds them after tmem_wait16.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
// Waits for this thread's TMEM loads; the values pass through the statement,
// so that no use of them can be scheduled before it.
__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

// Element k (0..15) of 16 register values, by a tree of selects on k's bits
// (no local memory).
__device__ __forceinline__ float select16(const uint32_t (&v)[16], int k) {
    float a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = __uint_as_float((k & 1) ? v[2 * i + 1] : v[2 * i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = (k & 2) ? a[2 * i + 1] : a[2 * i];
#pragma unroll
    for (int i = 0; i < 2; ++i) a[i] = (k & 4) ? a[2 * i + 1] : a[2 * i];
    return (k & 8) ? a[1] : a[0];
}

// Three-input minimum (sm_100 and later).
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Order-preserving encoding of a float key as an unsigned word.
__device__ __forceinline__ uint32_t key_enc(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_dec(uint32_t e) {
    return __uint_as_float((e & 0x80000000u) ? (e & 0x7FFFFFFFu) : ~e);
}

struct KnnArgs {
    int Dp;
    long long ntp;                    // point tiles of this pass
    int op_stages;
    int s32;                          // sample pass: chunks per segment
    unsigned int nd;                  // dense queries
    const KnnQuery* qinfo;            // [dense position]
    const float* qlim;                // [dense position] key limit of the full pass
    const float* w;                   // |x|^2 of the pass's points, FLT_MAX past the last
    float* smin;                      // sample pass: [Qcap][nws] smallest member key of each chunk
    int nws;
    uint2* part;                      // full pass: lists of (key, id), list_cap each
    int list_cap;
    int* part_n;
    int* err;
};

// The CTA whose range of (query tile, point tile) pairs holds pair p: ranges
// are [c U / G, (c + 1) U / G).
__device__ __forceinline__ int owner_cta(long long p, long long U, int G) {
    return (int)(((p + 1) * G - 1) / U);
}

// kSample: the sample pass (chunk minima), else the full pass (lists).
// kStream: D > kResidentD, query slabs travel with the point slabs.
template <bool kSample, bool kStream>
__global__ void __launch_bounds__(kKnnThreads, 1)
    k_knn_tc(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_x,
             const __grid_constant__ CUtensorMap tm_bm, KnnArgs a) {
    constexpr uint32_t kTmemCols = 2 * MH * BN;
    const unsigned int nd = a.nd;
    const long long nqt = ((long long)nd + MQ - 1) / MQ;
    const long long ntp = a.ntp;
    const long long U = nqt * ntp;
    const int G = (int)min((long long)gridDim.x, U);
    if ((int)blockIdx.x >= G) return;
    const long long p0 = (long long)blockIdx.x * U / G, p1 = (long long)(blockIdx.x + 1) * U / G;
    const int atoms = a.Dp / 64;
    const int apst = kStream ? 1 : atoms;   // 64-column slabs per operand stage
    const int nst = kStream ? atoms : 1;    // operand stages per tile
    const int ops = a.op_stages;

    extern __shared__ __align__(1024) unsigned char smraw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
    unsigned char* sQ = base;                                                  // resident query tile
    unsigned char* sOp = sQ + (kStream ? 0u : (uint32_t)atoms * kQSlab);       // ring: [points][queries if streamed]
    const uint32_t xbytes = (uint32_t)apst * kXSlab;
    const uint32_t op_stride = xbytes + (kStream ? kQSlab : 0u);
    unsigned char* sE = sOp + (size_t)ops * op_stride;                         // ring: [membership][norms]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sE + (size_t)kEpStages * kEpStride);
    uint64_t* a_full = bars;
    uint64_t* a_empty = bars + 1;
    uint64_t* tfull = bars + 2;                      // [accumulator set][half]
    uint64_t* tempty = tfull + 2 * MH;               // [accumulator set][half]
    uint64_t* done_bar = tempty + 2 * MH;
    uint64_t* full_op = done_bar + 1;                // [ops]
    uint64_t* empty_op = full_op + ops;              // [ops]
    uint64_t* full_ep = empty_op + ops;              // [kEpStages]
    uint64_t* empty_ep = full_ep + kEpStages;        // [kEpStages]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty_ep + kEpStages);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // known to be warp-uniform
    if (tid == 0) {
        bar_init(a_full, 1);
        bar_init(a_empty, MW);
        for (int s = 0; s < 2 * MH; ++s) {
            bar_init(tfull + s, 1);
            bar_init(tempty + s, KM / 32);
        }
        bar_init(done_bar, MW);
        for (int s = 0; s < ops; ++s) {
            bar_init(full_op + s, 1);
            bar_init(empty_op + s, MW);
        }
        for (int s = 0; s < kEpStages; ++s) {
            bar_init(full_ep + s, 1);
            bar_init(empty_ep + s, NEPI / NCH);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---- TMA producer ----
        long long cur_qt = -1;
        int j = -1;
        // (query tile, point tile) and both rings' stage and round parity,
        // advanced incrementally (no 64-bit division per tile)
        long long qt = p0 / ntp, pt = p0 - qt * ntp;
        int s = 0, e = 0;
        uint32_t spar = 0, epar = 0;
        long long issued_op = 0, issued_ep = 0;   // copies issued into each ring
        bool ok = true;
        for (long long p = p0; p < p1 && ok && !*abort_flag; ++p) {
            if (!kStream && qt != cur_qt) {
                ++j;
                cur_qt = qt;
                if (j >= 1 && !bar_wait(a_empty, (uint32_t)((j - 1) & 1), abort_flag, a.err)) break;
                bar_expect_tx(a_full, (uint32_t)atoms * kQSlab);
                for (int k = 0; k < atoms; ++k)
                    tma_2d(sQ + (size_t)k * kQSlab, &tm_q, a_full, k * 64, (int)(qt * MQ));
            }
            for (int sl = 0; sl < nst; ++sl) {
                if (issued_op >= ops && !bar_wait(empty_op + s, spar ^ 1u, abort_flag, a.err)) {
                    ok = false;
                    break;
                }
                unsigned char* xs = sOp + (size_t)s * op_stride;
                bar_expect_tx(full_op + s, op_stride);
                for (int k = 0; k < apst; ++k) {
                    const int col = (sl * apst + k) * 64;
                    if constexpr (kSample) {
                        // a tile is four chunks of 32 sample points
#pragma unroll
                        for (int i = 0; i < BN / 32; ++i) {
                            const int c = (int)(pt * (BN / 32)) + i;
                            const int seg = c / a.s32;
                            tma_4d(xs + (size_t)k * kXSlab + i * 32 * 128, &tm_x, full_op + s, col, c - seg * a.s32, 0,
                                   seg);
                        }
                    } else {
                        tma_2d(xs + (size_t)k * kXSlab, &tm_x, full_op + s, col, (int)(pt * BN));
                    }
                }
                if constexpr (kStream) tma_2d(xs + xbytes, &tm_q, full_op + s, sl * 64, (int)(qt * MQ));
                ++issued_op;
                if (++s == ops) { s = 0; spar ^= 1u; }
                if (sl == 0) {
                    if (issued_ep >= kEpStages && !bar_wait(empty_ep + e, epar ^ 1u, abort_flag, a.err)) {
                        ok = false;
                        break;
                    }
                    unsigned char* es = sE + (size_t)e * kEpStride;
                    bar_expect_tx(full_ep + e, kEpStride);
                    tma_2d(es, &tm_bm, full_ep + e, (int)(pt * BW), (int)(qt * MQ));
                    bulk_copy(es + kBmBytes, a.w + pt * BN, kWBytes, full_ep + e);
                    ++issued_ep;
                    if (++e == kEpStages) { e = 0; epar ^= 1u; }
                }
            }
            if (++pt == ntp) { pt = 0; ++qt; }
        }
        // Drain: every copy issued into a ring stage completes before exit.
        for (int st = 0; st < ops && st < issued_op; ++st) {
            const long long last = st + ((issued_op - 1 - st) / ops) * ops;
            bar_drain(full_op + st, (uint32_t)((last / ops) & 1), a.err);
        }
        for (int et = 0; et < kEpStages && et < issued_ep; ++et) {
            const long long last = et + ((issued_ep - 1 - et) / kEpStages) * kEpStages;
            bar_drain(full_ep + et, (uint32_t)((last / kEpStages) & 1), a.err);
        }
        if (j >= 0) bar_drain(a_full, (uint32_t)(j & 1), a.err);
    } else if (warp >= 1 && warp <= MW) {
        // ---- MMA issuers ----
        // One warp per half of the query tile: while one waits for a barrier
        // (a few hundred cycles even for a completed phase) the other's
        // products keep the tensor pipe busy. The whole warp walks the loop, so
        // that descriptors and counters are warp-uniform values; one elected
        // lane issues (a loop run by one lane alone moved every descriptor
        // through vector registers and issued one product in 178 cycles; the
        // pipe takes 64).
        // kind::f16: FP32 accumulator, fp16 A and B, both K-major, N = BN, M = 128.
        const int hq = warp - 1;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(KM >> 4) << 24);
        const uint64_t qdesc = desc_sw128(smem_addr(kStream ? sOp + xbytes : sQ) + (uint32_t)(hq * KM * 128));
        const uint64_t xdesc = desc_sw128(smem_addr(sOp));
        const bool leader = elect_one();
        long long cur_qt = -1;
        int j = -1;
        long long i = 0;
        long long qt = p0 / ntp, pt = p0 - qt * ntp;
        int s = 0;
        uint32_t spar = 0;
        bool ok = true;
        for (long long p = p0; p < p1 && ok; ++p, ++i) {
            if (!kStream && qt != cur_qt) {
                if (j >= 0 && leader) mma_commit(a_empty);
                ++j;
                cur_qt = qt;
                ok = __all_sync(0xffffffffu, bar_wait(a_full, (uint32_t)(j & 1), abort_flag, a.err));
                if (!ok) break;
            }
            const bool work = qt * MQ + hq * KM < (long long)nd;   // a half without queries is left out
            if (++pt == ntp) { pt = 0; ++qt; }
            const int acc = (int)(i & 1);
            const int ab = acc * MH + hq;
            ok = i < 2 || __all_sync(0xffffffffu, bar_wait(tempty + ab, (uint32_t)(((i >> 1) - 1) & 1), abort_flag, a.err));
            if (!ok) break;
            const uint32_t d = tmem + (uint32_t)(ab * BN);
            for (int sl = 0; sl < nst; ++sl) {
                ok = __all_sync(0xffffffffu, bar_wait(full_op + s, spar, abort_flag, a.err));
                if (!ok) break;
                fence_after();
                // descriptors advance by adding the byte offset / 16 to their
                // start-address field (shared addresses stay below 2^18: no carry)
                const uint64_t so = (uint64_t)(s * (op_stride >> 4));
                const uint64_t dx = xdesc + so, dq = kStream ? qdesc + so : qdesc;
                if (leader) {
                    if (work)
                        for (int at = 0; at < apst; ++at) {
                            const uint64_t da = dq + (uint64_t)((at * kQSlab) >> 4);
                            const uint64_t db = dx + (uint64_t)((at * kXSlab) >> 4);
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                mma_f16(d, da + (uint64_t)(ks * 2), db + (uint64_t)(ks * 2), idesc,
                                        (ks | at | sl) > 0 ? 1u : 0u);
                        }
                    mma_commit(empty_op + s);
                    if (sl + 1 == nst) mma_commit(tfull + ab);
                }
                __syncwarp();
                if (++s == ops) { s = 0; spar ^= 1u; }
            }
        }
        // every product has landed before TMEM is released
        if (leader) mma_commit(done_bar);
        __syncwarp();
    } else if (warp > MW) {
        // ---- epilogue ----
        // Eight warps per accumulator set, so that a warp visits every second
        // tile: the fixed cost of a visit (barrier waits, loads of the query's
        // membership) is paid once per 128 columns instead of once per 64, and
        // two tiles' epilogues overlap.
        const int ew = warp - 1 - MW;
        const int quad = warp & 3;                    // TMEM lanes this warp may read
        const int hq = (ew >> 2) % MH;                // query half (its own accumulator)
        const int acc = (ew >> 2) / MH;               // accumulator set, of tiles acc, acc + 2, ...
        const int ab = acc * MH + hq;
        const int row = hq * KM + quad * 32 + lane;   // query of the tile
        int n = 0;                                    // survivors in this lane's list
        uint2* list = nullptr;
        float m = 0.0f, lim = 0.0f;
        long long cur_qt = -1;
        auto close_list = [&](long long q) {
            a.part_n[(((long long)blockIdx.x + q) * NCH + acc) * MQ + row] = n;
        };
        long long qt = p0 / ntp, pt = p0 - qt * ntp;
        // A query tile can be crossed between this group's visits: its list is
        // opened (and closed, if empty) all the same.
        auto open_list = [&]() {
            if (!kSample && cur_qt >= 0) close_list(cur_qt);
            cur_qt = qt;
            n = 0;
            const int gq = (int)qt * MQ + row;   // dense position of this lane's query
            const bool live = (unsigned int)gq < nd;
            m = live ? (kSample ? a.qinfo[gq].m_up : a.qinfo[gq].m_lo) : 0.0f;
            if constexpr (!kSample) {
                lim = live ? a.qlim[gq] : -INFINITY;   // no key is below -infinity
                list = a.part + ((((long long)blockIdx.x + qt) * NCH + acc) * MQ + row) * a.list_cap;
            }
        };
        int e = 0;
        uint32_t epar = 0, tpar = 0;
        bool mine = acc == 0;
        for (long long p = p0; p < p1; ++p, mine = !mine) {
            if (qt != cur_qt) open_list();
            if (mine) {
                // every lane waits (and so sees the copied data); the warp leaves
                // together if any lane gave up, since tcgen05.ld is warp-wide
                const bool ok = bar_wait(full_ep + e, epar, abort_flag, a.err) &&
                                bar_wait(tfull + ab, tpar, abort_flag, a.err);
                if (!__all_sync(0xffffffffu, ok)) break;
                tpar ^= 1u;
                fence_after();
                const bool work = qt * MQ + hq * KM < (long long)nd;   // warp-uniform
                if (work) {
                    const unsigned char* es = sE + (size_t)e * kEpStride;
                    const uint4 mw = *reinterpret_cast<const uint4*>(es + (size_t)row * BW * 4);
                    const float* wv = reinterpret_cast<const float*>(es + kBmBytes);
                    const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(ab * BN);
                    // 16 columns at a time in two register sets: the next ones
                    // are loaded while these are examined. The accumulator goes
                    // back to the MMA warp as soon as the last ones are in
                    // registers.
                    uint32_t rc[2][16];
                    float mprev = INFINITY;   // sample pass: minimum of a chunk's first half
                    __syncwarp();   // tcgen05.ld is warp-collective
                    tmem_ld16(tbase, rc[0]);
#pragma unroll
                    for (int c = 0; c < BN / 16; ++c) {
                        uint32_t(&v)[16] = rc[c & 1];
                        tmem_wait16(v);
                        if (c + 1 < BN / 16) {
                            __syncwarp();
                            tmem_ld16(tbase + (uint32_t)((c + 1) * 16), rc[(c + 1) & 1]);
                        } else {
                            fence_before();
                            __syncwarp();
                            if (lane == 0) bar_arrive(tempty + ab);
                        }
                        // keys t = |x|^2 + m acc (packed FMA, in place)
#pragma unroll
                        for (int k = 0; k < 16; k += 4) {
                            const float4 w4 = *reinterpret_cast<const float4*>(wv + c * 16 + k);
                            const float2 a2 = __ffma2_rn(make_float2(m, m),
                                                         make_float2(__uint_as_float(v[k]), __uint_as_float(v[k + 1])),
                                                         make_float2(w4.x, w4.y));
                            const float2 b2 = __ffma2_rn(make_float2(m, m),
                                                         make_float2(__uint_as_float(v[k + 2]), __uint_as_float(v[k + 3])),
                                                         make_float2(w4.z, w4.w));
                            v[k] = __float_as_uint(a2.x);
                            v[k + 1] = __float_as_uint(a2.y);
                            v[k + 2] = __float_as_uint(b2.x);
                            v[k + 3] = __float_as_uint(b2.y);
                        }
                        const uint32_t word = c < 2 ? mw.x : c < 4 ? mw.y : c < 6 ? mw.z : mw.w;
                        const uint32_t mbits = (c & 1) ? word >> 16 : word & 0xFFFFu;
                        if constexpr (kSample) {
#pragma unroll
                            for (int k = 0; k < 16; ++k) v[k] = ((mbits >> k) & 1u) ? v[k] : 0x7f800000u;
                        }
                        float mm[5];
#pragma unroll
                        for (int k = 0; k < 5; ++k)
                            mm[k] = fmin3(__uint_as_float(v[3 * k]), __uint_as_float(v[3 * k + 1]),
                                          __uint_as_float(v[3 * k + 2]));
                        const float mn = fmin3(fmin3(mm[0], mm[1], mm[2]), fminf(mm[3], mm[4]), __uint_as_float(v[15]));
                        if constexpr (kSample) {
                            if (c & 1)
                                a.smin[(qt * MQ + row) * a.nws + pt * (BN / 32) + (c >> 1)] = fminf(mn, mprev);
                            else
                                mprev = mn;
                        } else if (mn < lim && mbits) {
                            const uint32_t id0 = (uint32_t)(pt * BN + c * 16);
                            uint32_t pm = 0;
#pragma unroll
                            for (int k = 0; k < 16; ++k) pm |= (__uint_as_float(v[k]) < lim ? 1u : 0u) << k;
                            for (pm &= mbits; pm; pm &= pm - 1) {
                                const int k = __ffs((int)pm) - 1;
                                if (n < a.list_cap)
                                    list[n] = make_uint2(__float_as_uint(select16(v, k)), id0 + (uint32_t)k);
                                ++n;   // a count above list_cap marks the list as overflowed
                            }
                        }
                    }
                } else {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(tempty + ab);
                }
                __syncwarp();
                if (lane == 0) bar_arrive(empty_ep + e);
            }
            if (++e == kEpStages) { e = 0; epar ^= 1u; }
            if (++pt == ntp) { pt = 0; ++qt; }
        }
        if (!kSample && cur_qt >= 0 && !*abort_flag) close_list(cur_qt);
    }
    if (warp == 1) bar_drain(done_bar, 0, a.err);   // both MMA warps' products
    __syncthreads();
    fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// Largest magnitude, value range and finiteness of the dataset.
__global__ void k_knn_scan(const float* __restrict__ X, int64_t n, KnnState* __restrict__ st) {
    int flags = 0, mneg = 0, mpos = 0;
    float amax = 0.0f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float x = __ldg(X + i);
        if (!(fabsf(x) <= FLT_MAX)) flags |= kKnnNonFinite;
        else amax = fmaxf(amax, fabsf(x));
        if (x == rintf(x) && fabsf(x) <= 256.0f) {
            mneg = max(mneg, 257 - (int)x);
            mpos = max(mpos, 257 + (int)x);
        } else {
            flags |= kKnnNotSmallInt;
        }
    }
    flags = __reduce_or_sync(0xffffffffu, flags);
    mneg = __reduce_max_sync(0xffffffffu, mneg);
    mpos = __reduce_max_sync(0xffffffffu, mpos);
    const uint32_t am = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));   // non-negative floats order as words
    if ((threadIdx.x & 31) == 0) {
        if (flags) atomicOr(&st->flags, flags);
        if (mneg) atomicMax(&st->mneg, mneg);
        if (mpos) atomicMax(&st->mpos, mpos);
        if (am) atomicMax(&st->amax, am);
    }
}

// Power-of-two scale that takes magnitudes up to amax below 2^15 (1 for zero).
__device__ __forceinline__ float knn_scale(float amax) {
    if (!(amax > 0.0f)) return 1.0f;
    return scalbnf(1.0f, 14 - ilogbf(amax));
}

// Shared row conversion of a warp: fp16(row * scale) into xh, the squared
// norm (RN) and the squared residual norm in scaled units (rounded up).
__device__ __forceinline__ void knn_row(const float* __restrict__ row, int D, int Dp, float scale, __half* xh, float& s,
                                        float& rr) {
    const int lane = threadIdx.x & 31;
    s = rr = 0.0f;
    for (int d = lane; d < Dp; d += 32) {
        const float x = d < D ? __ldg(row + d) : 0.0f;
        const float xs = x * scale;   // exact: a power of two, no overflow
        const __half h = __float2half_rn(xs);
        const float r = __fsub_rn(xs, __half2float(h));
        xh[d] = h;
        s = __fmaf_rn(x, x, s);
        rr = __fmaf_ru(r, r, rr);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
        rr = __fadd_ru(rr, __shfl_xor_sync(0xffffffffu, rr, o));
    }
}

// Residual that any row of D elements in scaled units may have beside the
// relative 2^-11 of its normal fp16 values (subnormals: half of 2^-24 each).
__device__ __forceinline__ float knn_abs_residual(int D) { return 1.01f * 2.98023224e-8f * sqrtf((float)D); }

// Dataset rows (once per index): fp16 operand, |x|^2 (FLT_MAX from row N up to
// the padded count) and the largest relative residual. One warp per row.
__global__ void k_knn_rows(const float* __restrict__ X, int64_t N, int D, int Dp, int64_t pad, __half* __restrict__ xh,
                           float* __restrict__ w, KnnState* __restrict__ st) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float scale = knn_scale(__uint_as_float(*(volatile uint32_t*)&st->amax));
    const float ar = knn_abs_residual(D);
    float rho = 0.0f;
    for (int64_t r = w0; r < pad; r += nw) {
        if (r >= N) {
            if (lane == 0) w[r] = FLT_MAX;
            continue;
        }
        float s, rr;
        knn_row(X + r * D, D, Dp, scale, xh + r * Dp, s, rr);
        // |x| scaled, rounded down; a zero row has no residual
        const float nx = sqrtf(s) * scale * 0.9999f, res = sqrtf(rr) * 1.0001f;
        if (res > ar && nx > 0.0f) rho = fmaxf(rho, (res - ar) / nx * 1.0001f);
        if (lane == 0) w[r] = s;
    }
    const uint32_t rm = __float_as_uint(rho);
    if (lane == 0 && rm) atomicMax(&st->rho, rm);
}

// Query rows of one search, in dense-list order (zero rows up to the next
// tile): fp16 operand, |q|^2, key multipliers and error terms. The norms of
// the sample points are gathered beside them. One warp per row.
__global__ void k_knn_qrows(KnnSearch k) {
    const int lane = threadIdx.x & 31;
    const int64_t g0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gn = (int64_t)gridDim.x * blockDim.x;
    if (k.f > 0) {
        const int64_t S = (int64_t)k.nseg * k.s32 * 32;
        for (int64_t j = g0; j < S; j += gn) {
            const int c = (int)(j >> 5), i = (int)(j & 31), seg = c / k.s32;
            k.w_sample[j] = k.w[(int64_t)seg * k.seg + ((int64_t)i * k.s32 + (c - seg * k.s32)) * k.f];
        }
    }
    const unsigned int nd = (unsigned int)k.nd;
    const int64_t npad = ((int64_t)nd + MQ - 1) / MQ * MQ;
    const KnnState ds = *k.dstate;
    const float sx = knn_scale(__uint_as_float(ds.amax));
    for (int64_t r = g0 >> 5; r < npad; r += gn >> 5) {
        __half* qh = static_cast<__half*>(k.qh) + r * k.Dp;
        if (r >= nd) {
            for (int d = lane; d < k.Dp; d += 32) qh[d] = __float2half_rn(0.0f);
            continue;
        }
        const float* row = k.queries + (int64_t)k.dense_q[r] * k.D;
        int bad = 0, mneg = 0, mpos = 0;
        float amax = 0.0f;
        for (int d = lane; d < k.D; d += 32) {
            const float x = __ldg(row + d);
            // beyond these magnitudes squares could leave the float range
            if (!(fabsf(x) <= kKnnMaxValue)) bad |= 2;
            else amax = fmaxf(amax, fabsf(x));
            if (x == rintf(x) && fabsf(x) <= 256.0f) {
                mneg = max(mneg, 257 - (int)x);
                mpos = max(mpos, 257 + (int)x);
            } else {
                bad |= 1;
            }
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        mneg = max(__reduce_max_sync(0xffffffffu, mneg), ds.mneg);
        mpos = max(__reduce_max_sync(0xffffffffu, mpos), ds.mpos);
        amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
        const bool unfit = (bad & 2) || (amax > 0.0f && amax < kKnnMinValue);
        const float sq = unfit ? 0.0f : knn_scale(amax);
        float s, rr;
        knn_row(row, k.D, k.Dp, sq, qh, s, rr);
        if (lane) continue;
        KnnQuery qi;
        qi.sq = s;
        if (unfit) {   // scanned exactly (k_knn_scan_rows); no survivors here
            qi = KnnQuery{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, kKnnUnfit};
            k.fallback[atomicAdd(k.n_fallback, 1u)] = (int)r;
        } else {
            const long long lo = 257 - mneg, hi = mpos - 257, mag = max(-lo, hi);
            const bool exact = !(ds.flags & kKnnNotSmallInt) && !bad && mneg > 0 && mpos > 0 &&
                               k.D * mag * mag < (1ll << 24) && k.D * (hi - lo) * (hi - lo) < (1ll << 24);
            const float m0 = -2.0f / (sq * sx);   // scales are powers of two
            if (exact) {
                qi.m_lo = qi.m_up = m0;
                qi.kappa = qi.slack = 0.0f;
                qi.flags = kKnnExact;
            } else {
                const float nq = sqrtf(s);
                const float rq = s > 0.0f ? sqrtf(rr) * 1.0001f / (sq * nq * 0.9999f) : 0.0f;
                qi.kappa = 1.01f * (rq + __uint_as_float(ds.rho)) + k.gamma;
                qi.slack = 2.02f * nq * (knn_abs_residual(k.D) / sx) + 1e-37f;
                qi.m_lo = m0 / (1.0f - qi.kappa);
                qi.m_up = m0 / (1.0f + qi.kappa);
                qi.flags = 0;
            }
        }
        k.qinfo[r] = qi;
        if (k.f == 0) k.qlim[r] = unfit ? -INFINITY : INFINITY;   // no sample pass
    }
}

// One warp: the bin of a 256-bin histogram that holds the want-th entry (in
// bin order, want >= 1) and the entry's rank within it. False when the bins
// hold fewer than want entries.
__device__ __forceinline__ bool select_bin(const uint32_t* hist, uint32_t want, uint32_t& bin, uint32_t& rest) {
    const int lane = threadIdx.x & 31;
    uint32_t mine = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) mine += hist[lane * 8 + b];
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    const uint32_t hit = __ballot_sync(0xffffffffu, x >= want);
    if (hit == 0) return false;
    const int src = __ffs((int)hit) - 1;
    uint32_t r = want - (x - mine), b = (uint32_t)lane * 8;
    if (lane == src)
        while (hist[b] < r) r -= hist[b++];
    bin = __shfl_sync(0xffffffffu, b, src);
    rest = __shfl_sync(0xffffffffu, r, src);
    return true;
}

constexpr int LW = 8;   // queries (warps) per block of k_knn_limit

// Key limit of each dense query's full pass from its chunk minima (one warp
// per query): the K-th smallest, then every key whose lower bound can reach its
// upper bound. The minima are read once, folded into 32 R groups held in
// registers (any K groups hold K different candidates; with at least 16 K
// groups two of the K nearest rarely share one), and the K-th smallest group
// is selected by radix passes over a 256-bin histogram, from the highest bit
// in which the groups differ (bits above it would send every lane to one bin).
// 10,000 queries of 1,953 chunks: 345 us with four passes over global memory
// from the top bit, 108 us from the first differing bit, 47 us from registers.
template <int R>
__global__ void __launch_bounds__(32 * LW) k_knn_limit(KnnSearch k) {
    __shared__ uint32_t hist[LW][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned int i = blockIdx.x * LW + w;
    if (i >= (unsigned int)k.nd) return;   // warps work alone
    const int nc = k.nws;
    const float* src = k.smin + (int64_t)i * nc;
    float v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = INFINITY;
    for (int c0 = 0; c0 < nc; c0 += 32 * R) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int c = c0 + j * 32 + lane;
            if (c < nc) v[j] = fminf(v[j], __ldg(src + c));
        }
    }
    uint32_t e[R], lo = 0xFFFFFFFFu, hi = 0, cnt = 0;   // encoded keys; range and count of the groups with a candidate
#pragma unroll
    for (int j = 0; j < R; ++j) {
        e[j] = v[j] < FLT_MAX ? key_enc(v[j]) : 0xFFFFFFFFu;
        if (e[j] != 0xFFFFFFFFu) {
            lo = min(lo, e[j]);
            hi = max(hi, e[j]);
            ++cnt;
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const KnnQuery q = k.qinfo[i];
    if (cnt < (uint32_t)k.K || (q.flags & kKnnUnfit)) {   // uniform: no limit, or no survivors
        if (lane == 0) k.qlim[i] = (q.flags & kKnnUnfit) ? -INFINITY : INFINITY;
        return;
    }
    uint32_t prefix = 0, want = (uint32_t)k.K;   // want-th smallest of e - lo with this prefix
    for (int top = 32 - __clz((int)(hi - lo)); top > 0;) {
        const int sh = max(top - 8, 0);
        for (int b = lane; b < 256; b += 32) hist[w][b] = 0;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t d = e[j] - lo;
            if (e[j] != 0xFFFFFFFFu && (top >= 32 ? 0u : d >> top) == prefix)
                atomicAdd(&hist[w][(d >> sh) & ((1u << (top - sh)) - 1u)], 1u);
        }
        __syncwarp();
        uint32_t bin = 0, rest = 0;
        select_bin(hist[w], want, bin, rest);
        prefix = (prefix << (top - sh)) | bin;
        want = rest;
        top = sh;
        __syncwarp();
    }
    if (lane) return;
    const float key = key_dec(lo + prefix);
    const double u = (1.0 + (double)q.kappa) * ((double)key + q.sq) + q.slack;
    const double l = (u + q.slack) / (1.0 - (double)q.kappa) - q.sq;
    // Keys below it survive: above every key that the bound admits, also where
    // all of its terms are zero (a zero query among zero points).
    k.qlim[i] = (float)(l + 1e-6 * (fabs(u) + q.sq) + 1e-37);
}

constexpr int MT = 128;   // threads of k_knn_merge

// Top-K of each dense query from its survivors (one block per query): step 3
// of the file comment. Survivors are (encoded key, id) words in shared memory;
// the chosen ones become (distance bits, id) words and are sorted.
__global__ void __launch_bounds__(MT) k_knn_merge(KnnSearch k) {
    extern __shared__ __align__(16) unsigned char msm[];
    unsigned long long* ent = reinterpret_cast<unsigned long long*>(msm);   // [kKnnMaxSurvivors]
    unsigned long long* sel = ent + kKnnMaxSurvivors;                       // [kKnnMaxChosen]
    float* qs = reinterpret_cast<float*>(sel + kKnnMaxChosen);              // [D]
    __shared__ uint32_t hist[256];
    __shared__ uint32_t s_cnt, s_bad, s_bin, s_rest, s_dmax, s_m, s_lo, s_hi;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned int nd = (unsigned int)k.nd;
    const int K = k.K, D = k.D;
    const long long ntp = ((long long)k.N + BN - 1) / BN;
    const long long U = (((long long)nd + MQ - 1) / MQ) * ntp;
    const int G = (int)min((long long)k.grid, U);
    const bool vec = (D & 3) == 0;
    for (unsigned int i = blockIdx.x; i < nd; i += gridDim.x) {
        const KnnQuery qi = k.qinfo[i];
        if (qi.flags & kKnnUnfit) continue;   // uniform
        const int q = k.dense_q[i];
        const long long qt = i / MQ;
        const int r = (int)(i - qt * MQ);
        const int c0 = owner_cta(qt * ntp, U, G), c1 = owner_cta(qt * ntp + ntp - 1, U, G);
        const int nl = (c1 - c0 + 1) * NCH;
        __syncthreads();
        if (tid == 0) {
            s_cnt = s_bad = s_dmax = s_m = s_hi = 0;
            s_lo = 0xFFFFFFFFu;
        }
        __syncthreads();
        // gather the lists: 16 lanes per list
        for (int l = tid >> 4; l < nl; l += MT / 16) {
            const long long lst = (((long long)(c0 + l / NCH) + qt) * NCH + l % NCH) * MQ + r;
            const int cnt = k.part_n[lst], have = min(cnt, k.list_cap);
            const uint2* src = k.part + lst * k.list_cap;
            uint32_t at = 0;
            if ((tid & 15) == 0) {
                at = atomicAdd(&s_cnt, (uint32_t)have);
                if (cnt > k.list_cap) s_bad = 1;
            }
            at = __shfl_sync(0xffffu << (lane & 16), at, lane & 16);
            for (int e = tid & 15; e < have; e += 16) {
                const uint2 v = src[e];
                if (at + e < (uint32_t)kKnnMaxSurvivors)
                    ent[at + e] = ((unsigned long long)key_enc(__uint_as_float(v.x)) << 32) | v.y;
            }
        }
        for (int d = tid; d < D; d += MT) qs[d] = k.queries[(int64_t)q * D + d];
        __syncthreads();
        const uint32_t n = s_cnt;
        if (s_bad) {   // uniform
            if (tid == 0) k.fallback[atomicAdd(k.n_fallback, 1u)] = (int)i;
            continue;
        }
        // every survivor, from shared memory or (more than it holds) the lists
        auto each = [&](auto f) {
            if (n <= (uint32_t)kKnnMaxSurvivors) {
                for (uint32_t e = tid; e < n; e += MT) f(ent[e]);
                return;
            }
            for (int l = tid >> 4; l < nl; l += MT / 16) {
                const long long lst = (((long long)(c0 + l / NCH) + qt) * NCH + l % NCH) * MQ + r;
                const int have = k.part_n[lst];
                const uint2* src = k.part + lst * k.list_cap;
                for (int e = tid & 15; e < have; e += 16) {
                    const uint2 v = src[e];
                    f(((unsigned long long)key_enc(__uint_as_float(v.x)) << 32) | v.y);
                }
            }
        };
        // K-th smallest encoded key (no limit when there are no more than K)
        uint32_t thr = 0xFFFFFFFFu;
        if (n > (uint32_t)K) {
            // digits from the highest bit in which the keys differ
            uint32_t lo = 0xFFFFFFFFu, hi = 0;
            each([&](unsigned long long v) {
                lo = min(lo, (uint32_t)(v >> 32));
                hi = max(hi, (uint32_t)(v >> 32));
            });
            __syncwarp();
            atomicMin(&s_lo, __reduce_min_sync(0xffffffffu, lo));
            atomicMax(&s_hi, __reduce_max_sync(0xffffffffu, hi));
            __syncthreads();
            lo = s_lo;
            uint32_t prefix = 0, want = (uint32_t)K;
            for (int top = 32 - __clz((int)(s_hi - lo)); top > 0;) {
                const int sh = max(top - 8, 0);
                for (int b = tid; b < 256; b += MT) hist[b] = 0;
                __syncthreads();
                each([&](unsigned long long w) {
                    const uint32_t v = (uint32_t)(w >> 32) - lo;
                    if ((top >= 32 ? 0u : v >> top) == prefix) atomicAdd(&hist[(v >> sh) & ((1u << (top - sh)) - 1u)], 1u);
                });
                __syncthreads();
                if (warp == 0) {
                    uint32_t bin = 0, rest = 0;
                    select_bin(hist, want, bin, rest);
                    if (lane == 0) {
                        s_bin = bin;
                        s_rest = rest;
                    }
                }
                __syncthreads();
                prefix = (prefix << (top - sh)) | s_bin;
                want = s_rest;
                top = sh;
            }
            thr = lo + prefix;
        }
        auto choose = [&](unsigned long long v) {
            const uint32_t at = atomicAdd(&s_m, 1u);
            if (at < (uint32_t)kKnnMaxChosen) sel[at] = v;
        };
        each([&](unsigned long long v) {
            if ((uint32_t)(v >> 32) <= thr) choose(v);
        });
        __syncthreads();
        uint32_t m = min(s_m, (uint32_t)kKnnMaxChosen);
        if (qi.flags & kKnnExact) {
            for (uint32_t e = tid; e < m; e += MT) {
                const float d = __fadd_rn(key_dec((uint32_t)(sel[e] >> 32)), qi.sq);
                sel[e] = ((unsigned long long)__float_as_uint(d) << 32) | (uint32_t)sel[e];
            }
        } else {
            // exact FP32 lane-order distances of sel[from, to): two lanes per
            // row (eight where D % 4 != 0)
            auto distances = [&](uint32_t from, uint32_t to) {
                const int per = vec ? 16 : 4, sub = vec ? lane >> 1 : lane >> 3;
                for (uint32_t b = from + warp * per; b < to; b += (MT / 32) * per) {
                    const uint32_t e = b + sub;
                    const bool on = e < to;
                    const uint32_t id = on ? (uint32_t)sel[e] : 0u;
                    const float d = row_distance(k.X + (int64_t)id * D, D, qs, vec, on);
                    __syncwarp();
                    if (on && (lane & (vec ? 1 : 7)) == 0) {
                        const uint32_t bits = d <= FLT_MAX ? __float_as_uint(d) : 0x7f800000u;   // NaN, inf: never listed
                        sel[e] = ((unsigned long long)bits << 32) | id;
                        atomicMax(&s_dmax, bits);
                    }
                }
            };
            distances(0, m);
            __syncthreads();
            if (n > (uint32_t)K) {
                // those K distances bound the K-th: the entries whose lower
                // bound they do not exclude
                const float top = __uint_as_float(s_dmax);
                each([&](unsigned long long v) {
                    const uint32_t ek = (uint32_t)(v >> 32);
                    if (ek <= thr) return;
                    const float low = __fsub_rd(__fmul_rd(1.0f - qi.kappa, __fadd_rd(key_dec(ek), qi.sq)), qi.slack);
                    if (low <= top) choose(v);
                });
                __syncthreads();
                const uint32_t m2 = min(s_m, (uint32_t)kKnnMaxChosen);
                distances(m, m2);
                m = m2;
            }
        }
        __syncthreads();
        if (s_m > (uint32_t)kKnnMaxChosen) {   // uniform
            if (tid == 0) k.fallback[atomicAdd(k.n_fallback, 1u)] = (int)i;
            continue;
        }
        // ascending (distance, id): bitonic over the next power of two
        uint32_t P = 32;
        while (P < m) P <<= 1;
        for (uint32_t e = m + tid; e < P; e += MT) sel[e] = ~0ull;
        __syncthreads();
        for (uint32_t a = 2; a <= P; a <<= 1)
            for (uint32_t b = a >> 1; b > 0; b >>= 1) {
                for (uint32_t t = tid; t < P / 2; t += MT) {
                    const uint32_t x = 2 * t - (t & (b - 1)), y = x + b;
                    const unsigned long long u = sel[x], v = sel[y];
                    if ((u > v) == ((x & a) == 0)) {
                        sel[x] = v;
                        sel[y] = u;
                    }
                }
                __syncthreads();
            }
        int32_t* oid = k.out_ids + (int64_t)q * K;
        float* od = k.out_d + (int64_t)q * K;
        for (int j = tid; j < K; j += MT) {
            const unsigned long long v = (uint32_t)j < m ? sel[j] : ~0ull;
            const bool have = (uint32_t)(v >> 32) < 0x7F7FFFFFu;   // finite, below FLT_MAX
            oid[j] = have ? (int32_t)(uint32_t)v : -1;
            od[j] = have ? __uint_as_float((uint32_t)(v >> 32)) : FLT_MAX;
        }
    }
}

// ---------------------------------------------------------------------------
// host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn knn_encode_fn() {
    static std::atomic<EncodeTiledFn> fn{nullptr};
    EncodeTiledFn f = fn.load();
    if (!f) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            f = reinterpret_cast<EncodeTiledFn>(p);
        fn = f;
    }
    return f;
}


// Map over an array of `rank` dimensions (strides in bytes, from the second).
bool knn_map(CUtensorMap* m, const void* ptr, CUtensorMapDataType dt, int rank, const cuuint64_t* dims,
             const cuuint64_t* strides, const cuuint32_t* box, bool swizzle) {
    EncodeTiledFn fn = knn_encode_fn();
    if (!fn) return false;
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, dt, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool knn_map_rows(CUtensorMap* m, const void* ptr, uint64_t cols, uint64_t rows, uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {2 * cols};
    const cuuint32_t box[2] = {64, box_rows};
    return knn_map(m, ptr, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, dims, strides, box, true);
}
bool knn_map_bits(CUtensorMap* m, const void* ptr, uint64_t words, uint64_t rows) {
    const cuuint64_t dims[2] = {words, rows}, strides[1] = {4 * words};
    const cuuint32_t box[2] = {BW, MQ};
    return knn_map(m, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, dims, strides, box, false);
}

size_t knn_smem(int Dp, int ops) {
    const size_t atoms = Dp / 64;
    const bool stream = Dp > kResidentD;
    const size_t op = stream ? kXSlab + kQSlab : atoms * kXSlab;
    return 1024 + (stream ? 0 : atoms * kQSlab) + ops * op + (size_t)kEpStages * kEpStride +
           8 * (3 + 4 * MH + 2 * ops + 2 * kEpStages) + 16;
}

template <bool kSample, bool kStream>
cudaError_t launch_knn_pass(const KnnSearch& k, cudaStream_t s) {
    static std::atomic<size_t> cap{0};
    const cudaError_t e = opt_in_smem(k_knn_tc<kSample, kStream>, k.smem, cap);
    if (e != cudaSuccess) return e;
    CUtensorMap mq, mx, mb;
    if (!knn_map_rows(&mq, k.qh, k.Dp, k.Qcap, MQ)) return cudaErrorNotSupported;
    KnnArgs a;
    a.Dp = k.Dp;
    a.op_stages = k.ops;
    a.s32 = k.s32;
    a.nd = (unsigned int)k.nd;
    a.qinfo = k.qinfo;
    a.qlim = k.qlim;
    a.smin = k.smin;
    a.nws = k.nws;
    a.part = k.part;
    a.list_cap = k.list_cap;
    a.part_n = k.part_n;
    a.err = k.err;
    if (kSample) {
        // sample point (segment g, chunk c, i) is row g seg + (i s32 + c) f
        const uint64_t row = 2 * (uint64_t)k.Dp;
        const cuuint64_t dims[4] = {(cuuint64_t)k.Dp, (cuuint64_t)k.s32, 32, (cuuint64_t)k.nseg};
        const cuuint64_t strides[3] = {(cuuint64_t)k.f * row, (cuuint64_t)k.s32 * k.f * row, (cuuint64_t)k.seg * row};
        const cuuint32_t box[4] = {64, 1, 32, 1};
        if (!knn_map(&mx, k.xh, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, dims, strides, box, true) ||
            !knn_map_bits(&mb, k.bm_sample, k.nws, k.Qcap))
            return cudaErrorNotSupported;
        a.ntp = (long long)k.nseg * k.s32 / (BN / 32);
        a.w = k.w_sample;
    } else {
        if (!knn_map_rows(&mx, k.xh, k.Dp, k.N, BN) || !knn_map_bits(&mb, k.bm, k.nwp, k.Qcap))
            return cudaErrorNotSupported;
        a.ntp = ((long long)k.N + BN - 1) / BN;
        a.w = k.w;
    }
    k_knn_tc<kSample, kStream><<<k.grid, kKnnThreads, k.smem, s>>>(mq, mx, mb, a);
    return cudaGetLastError();
}

size_t merge_smem(int D) { return 8 * (size_t)(kKnnMaxSurvivors + kKnnMaxChosen) + 4 * (size_t)D; }

}  // namespace

float knn_gamma(int D) {
    // accumulation of D products (one 2^-23 step per summed product), norms
    // and key arithmetic ((D + 16) + 8 roundings), the exact distance's own
    // FP32 lane order (gamma_n, n = ceil(D/8) + 6, twice: d <= 2 S); all with
    // margins.
    const double u = std::ldexp(1.0, -24), nn = (double)((D + 7) / 8 + 6);
    const double gn = nn * u / (1.0 - nn * u);
    return std::nextafter((float)(1.1 * (1.25 * (D + 16) * 2.0 * u + 2.0 * gn + (D + 24) * u)), INFINITY);
}

bool knn_plan(KnnSearch& k, int max_smem, size_t bitmap_smem) {
    if (k.D < 1 || k.D > kMaxKnnD || k.K < 1 || k.K > kMaxKnnK || k.N < 1) return false;
    // A sample of N / f points bounds the K-th distance when it has at least
    // 3 K chunks of 32; below 128 K points even the whole dataset is too coarse
    // a sample, and without a limit every candidate survives: allowed only
    // where all of them fit the merge.
    if (k.N < 128ll * k.K && k.N > kKnnMaxSurvivors) return false;
    k.Dp = (k.D + 63) / 64 * 64;
    k.ops = 0;
    for (int ops = kMaxOpStages; ops >= 2 && !k.ops; --ops)
        if (knn_smem(k.Dp, ops) <= (size_t)max_smem) {
            k.ops = ops;
            k.smem = knn_smem(k.Dp, ops);
        }
    if (!k.ops) return false;
    k.nwp = (int)((((int64_t)k.N + 31) / 32 + 3) / 4 * 4);
    k.f = 0;
    if (k.N >= 128ll * k.K) {
        // survivors are about f K: 1,024 of them at most, and a sixteenth of
        // the points (6 % more tensor work) is enough for any K up to 64
        k.f = 16;
        while (k.f > 1 && (k.f * k.K > 1024 || k.N / (32ll * k.f) < 3ll * k.K)) k.f >>= 1;
    }
    // segments of the membership kernel: as few as fit a block's bitmap (the
    // last one also takes what rounding leaves over)
    const int step = 128 * std::max(k.f, 1);
    const int64_t bits = (int64_t)bitmap_smem * 8 - 128;
    if (bits < 4 * step) return false;
    for (k.nseg = 1;; ++k.nseg) {
        k.seg = (int)((int64_t)k.N / k.nseg / step * step);
        if ((int64_t)k.N - (int64_t)(k.nseg - 1) * k.seg <= bits) break;
    }
    if (k.seg == 0) {   // fewer points than a sample step: one segment, no sample
        k.seg = k.N;
        k.f = 0;
    }
    k.s32 = k.f ? k.seg / (32 * k.f) : 0;
    k.nws = k.nseg * k.s32;
    // List capacity: within 512 MB of lists, at least 64 entries, never more
    // than a CTA's range can hold. CULSH_KNN_LIST_MARGIN sets it to K plus a
    // margin (the tests use 0 to reach the exact scan).
    const int64_t ntp = ((int64_t)k.N + BN - 1) / BN, nqt = k.Qcap / MQ;
    const int64_t sets = std::min<int64_t>(k.grid, nqt * ntp) + nqt;
    int64_t lc = std::min<int64_t>(1024, (int64_t(512) << 20) / (8 * sets * NT));
    lc = std::min<int64_t>(std::max<int64_t>(lc, 64), BN * (nqt * ntp / k.grid / NCH + 2));
    if (const char* e = getenv("CULSH_KNN_LIST_MARGIN")) lc = k.K + std::max(0, atoi(e));
    k.list_cap = (int)lc;
    return true;
}

size_t knn_part_lists(const KnnSearch& k) {
    const int64_t ntp = ((int64_t)k.N + BN - 1) / BN, nqt = k.Qcap / MQ;
    return (size_t)(std::min<int64_t>(k.grid, nqt * ntp) + nqt) * NT;
}
size_t knn_part_entries(const KnnSearch& k) { return knn_part_lists(k) * (size_t)k.list_cap; }

cudaError_t launch_knn_rows_dataset(const float* X, int64_t N, int D, int Dp, void* xh, float* w, int64_t pad,
                                    KnnState* st, cudaStream_t s) {
    const int64_t n = N * D;
    k_knn_scan<<<(unsigned)std::min<int64_t>((n + 1023) / 1024, 152 * 16), 256, 0, s>>>(X, n, st);
    const int blocks = (int)std::min<int64_t>((pad * 32 + 255) / 256, 152 * 16);
    k_knn_rows<<<blocks, 256, 0, s>>>(X, N, D, Dp, pad, static_cast<__half*>(xh), w, st);
    return cudaGetLastError();
}

int knn_launches(const KnnSearch& k) { return k.f > 0 ? 5 : 3; }

cudaError_t launch_knn_search(const KnnSearch& k, cudaStream_t s) {
    const int qblocks = (int)std::min<int64_t>(((int64_t)k.Qcap * 32 + 255) / 256, 152 * 8);
    k_knn_qrows<<<qblocks, 256, 0, s>>>(k);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const bool stream = k.Dp > kResidentD;
    if (k.f > 0) {
        e = stream ? launch_knn_pass<true, true>(k, s) : launch_knn_pass<true, false>(k, s);
        if (e != cudaSuccess) return e;
        const unsigned lb = (unsigned)((k.Qcap + LW - 1) / LW);
        if (k.K <= 64) k_knn_limit<32><<<lb, 32 * LW, 0, s>>>(k);
        else if (k.K <= 128) k_knn_limit<64><<<lb, 32 * LW, 0, s>>>(k);
        else k_knn_limit<128><<<lb, 32 * LW, 0, s>>>(k);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    e = stream ? launch_knn_pass<false, true>(k, s) : launch_knn_pass<false, false>(k, s);
    if (e != cudaSuccess) return e;
    static std::atomic<size_t> cap{0};
    const size_t smem = merge_smem(k.D);
    if ((e = opt_in_smem(k_knn_merge, smem, cap)) != cudaSuccess) return e;
    k_knn_merge<<<(unsigned)std::min<int64_t>(k.Qcap, 152 * 16), MT, smem, s>>>(k);
    return cudaGetLastError();
}

}  // namespace culsh
