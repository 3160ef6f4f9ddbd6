// K1 on the 5th-generation tensor cores (tcgen05 + TMA + TMEM).
//
// Replaces, for index builds, the per-table cublasSgemm + -b + /W + floor of
// cuLSH_Indexing.cu:27-66 and cuLSH_Kernels.cu:40-101 with one persistent
// GEMM over all L*M columns whose epilogue produces the exact canonical FP32
// bucket codes.
//
// Exactness. X and A are scaled by powers of two (the largest magnitude of a
// sample of X, of all of A, goes to 2^10) and split into fp16 parts, X = Xh + Xl
// and A = Ah + Al (Xl is skipped when every element is exact in fp16). The
// tensor cores compute y = Xh*Al' (+ Xl*Ah') + Xh*Ah' with FP32 accumulation
// in TMEM, the small products first. For each element the distance between y
// and the canonical sequential FMA chain is bounded by E = kappa * |x|_t * |a|_t, where
// kappa covers the split residue (2^-22 per part: fp16 pairs keep 22 bits, bf16
// pairs had kept 16), a rounding at every accumulation of the large products
// (one 2^-23 step per product; the small ones accumulate at 2^-11 of that) and
// the canonical chain's own rounding (D + 2 steps of 2^-24), with a 1.25 margin.
// Both sums run over d in order, so a rounding is relative to the sum so far,
// which Cauchy-Schwarz bounds by the norms of x's and a's leading parts: an
// element takes part in the roundings from its own 16-wide step on. Summed over
// the steps (Cauchy-Schwarz again) that is the product of the weighted norms
// |x|_t = sqrt(sum t_d x_d^2), t_d = 1 - slope * (d rounded down to 16), where
// slope * D is the share of kappa that such roundings have. A window
// test on (y - b) * (1/W) without a division proves a code: when no integer
// lies within E / W and the test's own rounding of it, every value the
// canonical chain can take has the same floor. Every other element is
// appended to a list and recomputed in the canonical order by k_tc_recompute.
// Codes are therefore bit-identical to the SIMT kernel and the oracle. With
// bf16 parts in any order 3.8 % of the codes of 1M x 128 integer features at
// W = 16 were open (0.69 ms of recomputation), with fp16 parts and plain norms
// 1.7 % (0.35 ms), now 1.0 % (0.22 ms).
//
// Structure: persistent CTAs of 18 warps. Warp 0 issues TMA loads (the
// projection matrix once, then 128-point X tiles into a 1- or 2-stage ring);
// warp 1 owns TMEM and issues tcgen05.mma (M=128, N=L*M padded to 16, K=16
// per instruction, fp16 inputs, FP32 accumulators, two accumulators so that
// the epilogue of one tile overlaps the MMAs of the next); warps 2-17 read
// TMEM with tcgen05.ld (four warps per lane quadrant, each taking a quarter
// of the columns) and run the epilogue. Codes the bound leaves open are appended
// row by row to a per-CTA list. Every mbarrier wait is bounded:
// on timeout the kernel raises kErrSpin and the host falls back to the SIMT
// kernel.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <climits>

#include "culsh_internal.cuh"

namespace culsh {
namespace {

constexpr int TC_M = 128;
constexpr int TC_EPI_WARPS = 16;                      // four per TMEM lane quadrant
constexpr int TC_THREADS = 64 + 32 * TC_EPI_WARPS;    // TMA warp, MMA warp, epilogue
constexpr uint32_t kPollLimit = 1u << 26;

struct TcArgs {
    int64_t N;
    int D, Dp, LM, LMp, ntiles, need_lo, stages, tmem_cols;
    float W, kappa;
    const float* b;        // [LM]
    const float* anorm;    // [LM] upper bounds of |a_c|_t
    const float* xnorm;    // [N]  upper bounds of |x_n|_t
    const ProjectState* ps;   // scales of X and A
    int32_t* codes;        // [LM][N]
    int32_t* pmin;         // [gridDim.x][LM]
    int32_t* pmax;
    unsigned long long* relist;   // (n << 16) | c of codes to recompute, one region per CTA
    unsigned long long relist_cap;        // entries per CTA region
    unsigned int* relist_cnt;             // [gridDim.x] entries used per region (may exceed the cap)
    int* err;
    uint32_t b_bytes, x_bytes;    // one fp16 operand region of A (LMp x Dp) / of an X tile (128 x Dp)
    // Streaming form (A too large to keep in shared memory): this launch
    // covers columns [col0, col0 + LM) of LMtot; each ring stage holds one
    // 64-wide K slice of Xh (Xl) and of Ah, Al.
    int col0, LMtot;
    uint32_t stage_bytes;         // streaming: bytes of one ring stage
    uint32_t a_chunk;             // streaming: bytes of one A slice (LMp x 64 fp16)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// One lane of the (converged) warp, the same on every call.
__device__ __forceinline__ bool elect_lane() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
// Bounded wait for the completion of the phase with the given parity. The
// single-thread producer and MMA roles back off between polls so that their
// spinning does not take issue slots from the epilogue warps.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err,
                                          bool backoff = false) {
    if (mbar_test_wait(bar, parity)) return true;   // cheaper than a suspending wait when the phase is over
    for (uint32_t i = 0; i < kPollLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (backoff) __nanosleep(64);
    }
    *abort_flag = 1;
    atomicOr(err, kErrSpin);
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row
// groups 1024 bytes apart (stride byte offset), sm_100 descriptor version.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(
            d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// kStream = false: A resident in shared memory (Dp, LMp <= 256), X tiles
// ring-buffered. kStream = true: X and A both streamed in 64-wide K slices,
// for any Dp; a launch covers at most 256 columns. Same epilogue.
template <bool kStream>
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_project_tc(const __grid_constant__ CUtensorMap tm_xh, const __grid_constant__ CUtensorMap tm_xl,
                 const __grid_constant__ CUtensorMap tm_ah, const __grid_constant__ CUtensorMap tm_al, TcArgs a) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    // 1024-byte aligned operand regions (the swizzle atoms assume it).
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
    unsigned char* sAh = base;
    unsigned char* sAl = sAh + (kStream ? 0 : a.b_bytes);
    // resident: stage s = Xh at s*(1+need_lo)*x_bytes, Xl right after;
    // streaming: stage s = [Xh slice][Xl slice][Ah slice][Al slice]
    unsigned char* sX = kStream ? base : sAl + a.b_bytes;
    const uint32_t stage_bytes = kStream ? a.stage_bytes : a.x_bytes * (a.need_lo ? 2u : 1u);
    unsigned char* tail = sX + (size_t)a.stages * stage_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(tail);
    uint64_t* empty = full + 2;
    uint64_t* tfull = empty + 2;
    uint64_t* tempty = tfull + 2;
    uint64_t* bfull = tempty + 2;
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
    unsigned int* list_top = reinterpret_cast<unsigned int*>(tmem_ptr + 2);
    int32_t* cmin = reinterpret_cast<int32_t*>(tail + 96);   // 16-byte aligned, past the barriers
    int32_t* cmax = cmin + a.LMp;
    float* s_an = reinterpret_cast<float*>(cmax + a.LMp);     // |a_c|_t bounds / W
    float* s_bw = s_an + a.LMp;                                // -b_c / W
    float* s_win = s_bw + a.LMp;                               // the window test's own rounding beside |v|
    uint32_t* s_unsure = reinterpret_cast<uint32_t*>(s_win + a.LMp);   // [8 words][TC_EPI_WARPS * 32] per-thread masks

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // known to be warp-uniform
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
            mbar_init(tfull + s, 1);
            mbar_init(tempty + s, TC_EPI_WARPS);
        }
        mbar_init(bfull, 1);
        *abort_flag = 0;
        *list_top = a.relist_cnt[blockIdx.x];   // a column block's list goes on from the one before
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int c = tid; c < a.LMp; c += TC_THREADS) {
        cmin[c] = INT_MAX;
        cmax[c] = INT_MIN;
        const float inv_w = 1.0f / a.W, bc = c < a.LM ? __ldg(a.b + a.col0 + c) : 0.0f;
        s_an[c] = c < a.LM ? __fmul_ru(__ldg(a.anorm + a.col0 + c), inv_w * 1.0001f) : 0.0f;
        s_bw[c] = -bc * inv_w;
        s_win[c] = fabsf(bc * inv_w) * 4.8e-7f + 1.5e-7f;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)),
                     "r"((uint32_t)a.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;
    const int katoms = a.Dp / 64, ksteps = a.Dp / 16;

    if (kStream && warp == 0 && lane == 0) {
        // ---- TMA producer, streaming: every tile, every K slice of X and A ----
        const uint32_t xb = 16384u;   // one X slice: 128 rows x 128 bytes
        int i = 0;
        for (int tile = blockIdx.x; tile < a.ntiles && !*abort_flag; tile += gridDim.x) {
            for (int k = 0; k < katoms; ++k, ++i) {
                const int s = i % a.stages;
                if (i >= a.stages &&
                    !mbar_wait(empty + s, (uint32_t)((i / a.stages - 1) & 1), abort_flag, a.err, true))
                    break;
                unsigned char* st = sX + (size_t)s * stage_bytes;
                unsigned char* sa = st + xb * (a.need_lo ? 2u : 1u);
                mbar_expect_tx(full + s, stage_bytes);
                tma_load_2d(st, &tm_xh, full + s, k * 64, tile * TC_M);
                if (a.need_lo) tma_load_2d(st + xb, &tm_xl, full + s, k * 64, tile * TC_M);
                tma_load_2d(sa, &tm_ah, full + s, k * 64, a.col0);
                tma_load_2d(sa + a.a_chunk, &tm_al, full + s, k * 64, a.col0);
            }
        }
    } else if (kStream && warp == 1) {
        // ---- MMA issuer, streaming (the whole warp walks, one lane issues) ----
        // kind::f16 instruction descriptor: FP32 accumulator, fp16 A and B,
        // both K-major, N = LMp, M = 128.
        const uint32_t idesc = (1u << 4) | ((uint32_t)(a.LMp >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
        const uint32_t xb = 16384u;
        const bool leader = elect_lane();
        int i = 0, t = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < a.ntiles && ok; tile += gridDim.x, ++t) {
            const int acc = t & 1;
            ok = t < 2 || __all_sync(0xffffffffu, mbar_wait(tempty + acc, (uint32_t)(((t >> 1) - 1) & 1), abort_flag, a.err, true));
            if (!ok) break;
            const uint32_t d = tmem + (uint32_t)(acc * a.LMp);
            for (int k = 0; k < katoms; ++k, ++i) {
                const int s = i % a.stages;
                ok = __all_sync(0xffffffffu, mbar_wait(full + s, (uint32_t)((i / a.stages) & 1), abort_flag, a.err, true));
                if (!ok) break;
                tc_fence_after();
                const uint32_t xs = smem_u32(sX + (size_t)s * stage_bytes);
                const uint32_t as = xs + xb * (a.need_lo ? 2u : 1u);
                const uint64_t xh = sw128_desc(xs), xl = sw128_desc(xs + xb), ah = sw128_desc(as),
                               al = sw128_desc(as + a.a_chunk);
                if (leader) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        umma_f16(d, xh + ks * 2, al + ks * 2, idesc, (k > 0 || ks > 0) ? 1u : 0u);
                    if (a.need_lo)
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) umma_f16(d, xl + ks * 2, ah + ks * 2, idesc, 1u);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) umma_f16(d, xh + ks * 2, ah + ks * 2, idesc, 1u);
                    umma_commit(empty + s);
                    if (k + 1 == katoms) umma_commit(tfull + acc);
                }
                __syncwarp();
            }
        }
    } else if (!kStream && warp == 0 && lane == 0) {
        // ---- TMA producer ----
        mbar_expect_tx(bfull, 2 * a.b_bytes);
        for (int k = 0; k < katoms; ++k) {
            tma_load_2d(sAh + (size_t)k * a.LMp * 128, &tm_ah, bfull, k * 64, a.col0);
            tma_load_2d(sAl + (size_t)k * a.LMp * 128, &tm_al, bfull, k * 64, a.col0);
        }
        int i = 0;
        for (int tile = blockIdx.x; tile < a.ntiles && !*abort_flag; tile += gridDim.x, ++i) {
            const int s = i % a.stages;
            if (i >= a.stages && !mbar_wait(empty + s, (uint32_t)((i / a.stages - 1) & 1), abort_flag, a.err, true))
                break;
            unsigned char* xh = sX + (size_t)s * stage_bytes;
            mbar_expect_tx(full + s, stage_bytes);
            for (int k = 0; k < katoms; ++k) {
                tma_load_2d(xh + (size_t)k * TC_M * 128, &tm_xh, full + s, k * 64, tile * TC_M);
                if (a.need_lo) tma_load_2d(xh + a.x_bytes + (size_t)k * TC_M * 128, &tm_xl, full + s, k * 64, tile * TC_M);
            }
        }
    } else if (!kStream && warp == 1) {
        // ---- MMA issuer (the whole warp walks, one lane issues) ----
        const uint32_t idesc = (1u << 4) | ((uint32_t)(a.LMp >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
        const bool leader = elect_lane();
        const uint64_t ah = sw128_desc(smem_u32(sAh)), al = sw128_desc(smem_u32(sAl));
        const uint64_t x0 = sw128_desc(smem_u32(sX));
        bool ok = __all_sync(0xffffffffu, mbar_wait(bfull, 0, abort_flag, a.err, true));
        int i = 0;
        for (int tile = blockIdx.x; tile < a.ntiles && ok; tile += gridDim.x, ++i) {
            const int s = i % a.stages, acc = i & 1;
            ok = (i < 2 || __all_sync(0xffffffffu, mbar_wait(tempty + acc, (uint32_t)(((i >> 1) - 1) & 1), abort_flag, a.err, true))) &&
                 __all_sync(0xffffffffu, mbar_wait(full + s, (uint32_t)((i / a.stages) & 1), abort_flag, a.err, true));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(acc * a.LMp);
            const uint64_t xh = x0 + (uint64_t)(s * (stage_bytes >> 4)), xl = xh + (a.x_bytes >> 4);
            if (leader) {
                // the small products first: their sums round at 2^-11 of the total
                auto product = [&](uint64_t x, uint64_t c, bool first) {
                    for (int ka = 0; ka < katoms; ++ka) {
                        const uint64_t xo = x + (uint64_t)((ka * TC_M * 128) >> 4), co = c + (uint64_t)((ka * a.LMp * 128) >> 4);
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks)
                            umma_f16(d, xo + ks * 2, co + ks * 2, idesc, (first && (ka | ks) == 0) ? 0u : 1u);
                    }
                };
                product(xh, al, true);
                if (a.need_lo) product(xl, ah, false);
                product(xh, ah, false);
                umma_commit(empty + s);
                umma_commit(tfull + acc);
            }
            __syncwarp();
        }
    } else if (warp >= 2) {
        // ---- epilogue: TMEM -> proven codes, list of codes to recompute ----
        const int ew = warp - 2;
        const int quad = warp & 3;                 // TMEM lane quadrant this warp may access
        const int part = ew >> 2;                  // which quarter of the column chunks
        const int row = quad * 32 + lane;
        const int nchunk = (a.LM + 15) / 16;       // the last column block may hold fewer than LMp / 16
        const int ch0 = part * nchunk / 4, ch1 = (part + 1) * nchunk / 4;
        uint32_t* my_mask = s_unsure + ew * 32 + lane;   // word w at my_mask[w * TC_EPI_WARPS * 32]
        unsigned long long* region = a.relist + (unsigned long long)blockIdx.x * a.relist_cap;
        int i = 0;
        // v = (y - b) / W up to rounding: acc * k1 - b / W, k1 = 1 / (scales W)
        const float k1 = __fdiv_rn(1.0f, a.W) / (a.ps->sx * a.ps->sa);   // the scales are powers of two
        for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, ++i) {
            const int acc = i & 1;
            const bool ok = mbar_wait(tfull + acc, (uint32_t)((i >> 1) & 1), abort_flag, a.err);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const int64_t n = (int64_t)tile * TC_M + row;
            const bool valid = n < a.N;
            const float kx = __fmul_ru(a.kappa, valid ? __ldg(a.xnorm + n) : 0.0f);
            uint32_t nuns = 0;
            for (int ch = ch0; ch < ch1; ++ch) {
                const int c0 = ch * 16;
                uint32_t r[16];
                __syncwarp();
                tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * a.LMp + c0), r);
                int32_t* out = a.codes + (int64_t)(a.col0 + c0) * a.N + n;
                const int live = a.LM - c0;                // columns of this chunk that exist
                const uint32_t cols = live >= 16 ? 0xFFFFu : (1u << live) - 1u;
                uint32_t unsure = 0, wide = 0;
#pragma unroll
                for (int j4 = 0; j4 < 16; j4 += 4) {
                    const float4 an = *reinterpret_cast<const float4*>(s_an + c0 + j4);
                    const float4 bw = *reinterpret_cast<const float4*>(s_bw + c0 + j4);
                    const float4 wn = *reinterpret_cast<const float4*>(s_win + c0 + j4);
                    const int4 mn = *reinterpret_cast<const int4*>(cmin + c0 + j4);
                    const int4 mx = *reinterpret_cast<const int4*>(cmax + c0 + j4);
                    auto one = [&](int j, float ac, float bc, float wc, int lo, int hi) {
                        // The window test: va is within win of every canonical
                        // v of a sum in [y - E, y + E]; no integer in that
                        // window proves the code. (From |va| = 2^21 on win
                        // exceeds a half: codes near the int32 range stay open.)
                        const float va = __fmaf_rn(__uint_as_float(r[j]), k1, bc);
                        const float fa = floorf(va);
                        const float fr = va - fa;
                        const float win = __fmaf_ru(kx, ac, __fmaf_ru(fabsf(va), 4.8e-7f, wc));
                        const bool sure = fminf(fr, 1.0f - fr) > win;
                        const int32_t code = __float2int_rz(fa);
                        r[j] = (uint32_t)code;
                        unsure |= sure ? 0u : 1u << j;
                        wide |= code < lo || code > hi ? 1u << j : 0u;
                    };
                    one(j4, an.x, bw.x, wn.x, mn.x, mx.x);
                    one(j4 + 1, an.y, bw.y, wn.y, mn.y, mx.y);
                    one(j4 + 2, an.z, bw.z, wn.z, mn.z, mx.z);
                    one(j4 + 3, an.w, bw.w, wn.w, mn.w, mx.w);
                }
                unsure = valid ? unsure & cols : 0u;
                wide = valid ? wide & cols & ~unsure : 0u;
                if (valid) {   // open codes are written over by the recomputation
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j < live) *out = (int32_t)r[j];
                        out += a.N;
                    }
                }
                // Column ranges: only columns with a code outside the range seen
                // so far reduce theirs (a warp reduction per column and value
                // for every chunk had taken most of the kernel: 0.61 ms at
                // 1M x 192 columns, now 0.32 ms).
                for (uint32_t m = __reduce_or_sync(0xffffffffu, wide); m; m &= m - 1) {
                    const int j = __ffs((int)m) - 1;
                    int32_t code = 0;
#pragma unroll
                    for (int k = 0; k < 16; ++k) code = k == j ? (int32_t)r[k] : code;
                    const bool use = (wide >> j) & 1u;
                    const int32_t lo = __reduce_min_sync(0xffffffffu, use ? code : INT_MAX);
                    const int32_t hi = __reduce_max_sync(0xffffffffu, use ? code : INT_MIN);
                    if (lane == 0) {
                        atomicMin(cmin + c0 + j, lo);
                        atomicMax(cmax + c0 + j, hi);
                    }
                }
                // bit (ch - ch0) * 16 + j of this thread's mask words
                const int w = (ch - ch0) >> 1;
                const uint32_t bits = unsure << (((ch - ch0) & 1) * 16);
                if (((ch - ch0) & 1) == 0) my_mask[w * TC_EPI_WARPS * 32] = bits;
                else my_mask[w * TC_EPI_WARPS * 32] |= bits;
                nuns += __popc(unsure);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty + acc);
            // Append this row's unsure columns contiguously (one atomic per warp).
            uint32_t incl = nuns;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if (total) {
                unsigned int basei = 0;
                if (lane == 31) basei = atomicAdd(list_top, total);
                basei = __shfl_sync(0xffffffffu, basei, 31);
                unsigned long long pos = (unsigned long long)basei + incl - nuns;
                const int nwords = (ch1 - ch0 + 1) >> 1;
                for (int w = 0; w < nwords && nuns; ++w) {
                    for (uint32_t m = my_mask[w * TC_EPI_WARPS * 32]; m; m &= m - 1) {
                        const int c = a.col0 + ch0 * 16 + w * 32 + (__ffs(m) - 1);
                        if (pos < a.relist_cap) region[pos] = ((unsigned long long)n << 16) | (unsigned)c;
                        ++pos;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int c = tid; c < a.LM; c += TC_THREADS) {
        a.pmin[(int64_t)blockIdx.x * a.LMtot + a.col0 + c] = cmin[c];
        a.pmax[(int64_t)blockIdx.x * a.LMtot + a.col0 + c] = cmax[c];
    }
    if (tid == 0) a.relist_cnt[blockIdx.x] = *list_top;
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols)
                     : "memory");
    }
}

// Power-of-two scale that takes magnitudes up to amax below 2^11 (1 for zero).
__device__ __forceinline__ float project_scale(uint32_t amax_bits) {
    const float amax = __uint_as_float(amax_bits);
    return amax > 0.0f ? scalbnf(1.0f, 10 - ilogbf(amax)) : 1.0f;
}

// A row (or column of A) of a warp: fp16 parts of row * scale into h and l
// (either may be null) and its squared weighted norm (t_d = 1 - slope * (d
// rounded down to 16)), rounded up. Lanes hold four consecutive elements where
// vec (16-byte aligned rows), one otherwise.
__device__ __forceinline__ void split_row(const float* __restrict__ row, int D, int Dp, float scale, float slope,
                                          bool vec, __half* h, __half* l, float& ss, bool& inexact, float& amax,
                                          bool& bad) {
    const int lane = threadIdx.x & 31;
    ss = 0.0f;
    auto part = [&](float x, float t, __half& hi, __half& lo) {
        const float xs = x * scale;   // exact but for subnormal results
        hi = __float2half_rn(xs);
        lo = __float2half_rn(__fsub_rn(xs, __half2float(hi)));
        inexact |= (__half_as_ushort(lo) & 0x7FFF) != 0;
        if (fabsf(x) <= FLT_MAX) amax = fmaxf(amax, fabsf(x));
        else bad = true;
        ss = __fmaf_ru(__fmul_ru(fabsf(x), t), fabsf(x), ss);
    };
    if (vec) {
        for (int d = 4 * lane; d < Dp; d += 128) {
            const float4 x = d < D ? __ldg(reinterpret_cast<const float4*>(row + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
            __align__(8) __half hh[4], ll[4];
            const float t = __fmaf_ru(-slope, (float)(d & ~15), 1.0f);
            part(x.x, t, hh[0], ll[0]);
            part(x.y, t, hh[1], ll[1]);
            part(x.z, t, hh[2], ll[2]);
            part(x.w, t, hh[3], ll[3]);
            if (h) *reinterpret_cast<uint2*>(h + d) = *reinterpret_cast<const uint2*>(hh);
            if (l) *reinterpret_cast<uint2*>(l + d) = *reinterpret_cast<const uint2*>(ll);
        }
    } else {
        for (int d = lane; d < Dp; d += 32) {
            __half hh, ll;
            part(d < D ? __ldg(row + d) : 0.0f, __fmaf_ru(-slope, (float)(d & ~15), 1.0f), hh, ll);
            if (h) h[d] = hh;
            if (l) l[d] = ll;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss = __fadd_ru(ss, __shfl_xor_sync(0xffffffffu, ss, o));
}

__device__ __forceinline__ float norm_up(float ss) { return __fmul_ru(__fsqrt_ru(ss), 1.00001f); }

// Norms of A's columns and of ns rows spread over X, the largest magnitudes of
// both (one warp per row); flag 8: some of those rows are not exact in fp16.
__global__ void k_project_sample(const float* __restrict__ X, int64_t N, int D, int ns, const float* __restrict__ A,
                                 int LM, float slope, float* __restrict__ xs, float* __restrict__ anorm,
                                 ProjectState* st) {
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (w >= ns + LM) return;
    const bool is_a = w >= ns;
    const float* row = is_a ? A + (int64_t)(w - ns) * D : X + (int64_t)w * (N / ns) * D;
    float ss, amax = 0.0f;
    bool inexact = false, bad = false;
    split_row(row, D, D, 1.0f, slope, false, nullptr, nullptr, ss, inexact, amax, bad);
    const uint32_t am = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    inexact = __any_sync(0xffffffffu, inexact);
    if (lane == 0) {
        if (!is_a && inexact) atomicOr(&st->flags, 8);
        (is_a ? anorm[w - ns] : xs[w]) = norm_up(ss);
        atomicMax(is_a ? &st->amax_a : &st->amax_x, am);
    }
}

// Scales from the largest magnitudes (run again after a conversion that the
// sample's scale took out of the fp16 range: amax_x is then X's own maximum).
__global__ void k_project_scales(ProjectState* st) {
    st->sx = project_scale(st->amax_x);
    st->sa = project_scale(st->amax_a);
}

// What an element's subnormal parts leave out (2^-25 of the scaled values, D of
// them against the other operand's plain norm, which is at most |.|_t over the
// root of the smallest weight), as an addition to |.|_t.
__device__ __forceinline__ float subnormal_residue(int D, float scale, float kappa, float slope) {
    return 1.01f * 2.98023224e-8f * sqrtf((float)D) / (scale * kappa * sqrtf(1.0f - slope * (float)D));
}

// fp16 parts of A (LMp rows, zero past LM) and upper bounds of its columns'
// weighted norms.
__global__ void k_split_a(const float* __restrict__ A, int LM, int LMp, int D, int Dp, float kappa, float slope, __half* ah,
                          __half* al, float* anorm, const ProjectState* st) {
    const int lane = threadIdx.x & 31;
    const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (c >= LMp) return;
    float ss, amax = 0.0f;
    bool inexact = false, bad = false;
    // rows past LM: zero dimensions to read
    split_row(A + (int64_t)min(c, LM - 1) * D, c < LM ? D : 0, Dp, st->sa, slope, false, ah + (int64_t)c * Dp,
              al + (int64_t)c * Dp, ss, inexact, amax, bad);
    if (lane == 0 && c < LM) anorm[c] = __fadd_ru(norm_up(ss), subnormal_residue(D, st->sa, kappa, slope));
}

// fp16 parts of X and upper bounds of its rows' weighted norms (warp per row); xl is null
// where the sample was exact in fp16. flags: 1 some element has a low part, 2
// a value is not finite, 4 a scaled value leaves the fp16 range (amax_x then
// holds the largest magnitude).
__global__ void k_split_rows(const float* __restrict__ X, int64_t N, int D, int Dp, float kappa, float slope,
                             __half* __restrict__ xh, __half* __restrict__ xl, float* __restrict__ xnorm, ProjectState* st) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float sx = st->sx, res = subnormal_residue(D, sx, kappa, slope);
    const bool vec = (D & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    float amax = 0.0f;
    bool inexact = false, bad = false;
    for (int64_t n = w0; n < N; n += nw) {
        float ss;
        split_row(X + n * D, D, Dp, sx, slope, vec, xh + n * Dp, xl ? xl + n * Dp : nullptr, ss, inexact, amax, bad);
        if (lane == 0) xnorm[n] = __fadd_ru(norm_up(ss), res);
    }
    const uint32_t am = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    const int f = (__any_sync(0xffffffffu, inexact) ? 1 : 0) | (__any_sync(0xffffffffu, bad) ? 2 : 0) |
                  (__uint_as_float(am) * sx > 65000.0f ? 4 : 0);
    if (lane == 0) {
        if (f & ~st->flags) atomicOr(&st->flags, f);
        if (f & 4) atomicMax(&st->amax_x, am);
    }
}

// Canonical-order recomputation of the codes the tensor-core bound could not
// prove (one thread per list entry; entries of CTA region r are
// list[r * cap .. r * cap + cnt[r])). A warp's 32 rows of X are fetched together,
// RD dimensions at a time: four (RD = 16) consecutive lanes read one row's 16-byte
// pieces, so that a load covers eight rows' 64 bytes instead of one 16-byte
// piece of 32 rows (which had bound the kernel on L1 lookups: 0.52 ms for 2.9M
// codes of 128 dimensions, now 0.34 ms); each lane then takes its own row
// from shared memory. A is staged there too where it fits (stage_a), with rows
// padded to D + 4 floats so that different columns at the same d spread over
// the banks.
constexpr int RT = 1024;       // threads
constexpr int RD = 16;         // dimensions per step
constexpr int RP = RD + 4;     // padded row
__global__ void __launch_bounds__(RT, 1) k_tc_recompute(const float* __restrict__ X, int64_t N, int D,
                               const float* __restrict__ A, const float* __restrict__ b, float W,
                               const unsigned long long* __restrict__ list, unsigned long long cap,
                               const unsigned int* __restrict__ cnt, int regions, int LM, int stage_a, int stage_x,
                               int32_t* __restrict__ codes, int32_t* __restrict__ cmin, int32_t* __restrict__ cmax,
                               int* __restrict__ err) {
    extern __shared__ __align__(16) float sX[];   // [warps][32][RP], then A
    __shared__ int32_t smin[1024], smax[1024];    // per-column ranges of this block (LM <= 1024 here)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* wx = sX + (size_t)warp * 32 * RP;
    float* sA = sX + (stage_x ? (size_t)(RT / 32) * 32 * RP : 0);
    const int Dq = (D & 3) == 0 ? D + 4 : D + 1;
    const bool block_range = LM <= 1024;
    if (block_range)
        for (int c = tid; c < LM; c += RT) {
            smin[c] = INT_MAX;
            smax[c] = INT_MIN;
        }
    if (stage_a)
        for (int i = tid; i < LM * D; i += RT) sA[(i / D) * Dq + (i % D)] = __ldg(A + i);
    __syncthreads();
    for (int r = blockIdx.x; r < regions; r += gridDim.x) {
        const unsigned int nr = min((unsigned long long)__ldg(cnt + r), cap);
        for (unsigned int k0 = warp * 32; k0 < nr; k0 += RT) {
            const bool on = k0 + lane < nr;
            const unsigned long long e = on ? list[(unsigned long long)r * cap + k0 + lane] : 0ull;
            const int64_t n = (int64_t)(e >> 16);
            const int c = (int)(e & 0xFFFF);
            const float* av = stage_a ? sA + (int64_t)c * Dq : A + (int64_t)c * D;
            float acc = 0.0f;
            if (stage_x) {
                for (int d0 = 0; d0 < D; d0 += RD) {
                    const int dl = d0 + 4 * (lane & 3);
                    float4 v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int64_t rn = __shfl_sync(0xffffffffu, n, i * 8 + (lane >> 2));
                        v[i] = dl < D ? __ldg(reinterpret_cast<const float4*>(X + rn * D + dl)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<float4*>(wx + (i * 8 + (lane >> 2)) * RP + 4 * (lane & 3)) = v[i];
                    __syncwarp();
                    const int dn = min(RD, D - d0);
#pragma unroll
                    for (int d = 0; d < RD; d += 4) {
                        if (d >= dn) break;   // uniform; D % 4 == 0 here
                        const float4 x4 = *reinterpret_cast<const float4*>(wx + lane * RP + d);
                        const float4 a4 = *reinterpret_cast<const float4*>(av + d0 + d);
                        acc = __fmaf_rn(x4.x, a4.x, acc);
                        acc = __fmaf_rn(x4.y, a4.y, acc);
                        acc = __fmaf_rn(x4.z, a4.z, acc);
                        acc = __fmaf_rn(x4.w, a4.w, acc);
                    }
                }
            } else if (on) {
                const float* x = X + n * D;
                for (int d = 0; d < D; ++d) acc = __fmaf_rn(__ldg(x + d), av[d], acc);
            }
            if (!on) continue;
            const float v = __fdiv_rn(__fsub_rn(acc, __ldg(b + c)), W);
            const float f = floorf(v);
            int32_t code = 0;
            if (!(fabsf(f) <= FLT_MAX)) atomicOr(err, kErrNonFinite);
            else if (!(f >= -2147483648.0f && f < 2147483648.0f)) atomicOr(err, kErrCodeRange);
            else code = (int32_t)f;
            codes[(int64_t)c * N + n] = code;
            if (block_range) {
                if (code < smin[c]) atomicMin(smin + c, code);
                if (code > smax[c]) atomicMax(smax + c, code);
            } else {
                atomicMin(cmin + c, code);
                atomicMax(cmax + c, code);
            }
        }
    }
    if (block_range) {
        __syncthreads();
        for (int c = tid; c < LM; c += RT) {
            if (smin[c] <= smax[c]) {
                atomicMin(cmin + c, smin[c]);
                atomicMax(cmax + c, smax[c]);
            }
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static std::atomic<EncodeTiledFn> fn{nullptr};
    EncodeTiledFn f = fn.load();
    if (!f) {   // several threads may look it up; all find the same
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

bool make_map(CUtensorMap* m, const void* ptr, uint64_t cols, uint64_t rows, uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

TcPlan tc_plan(int64_t N, int D, int LM, int num_sms, int max_smem) {
    TcPlan p{};
    p.Dp = (D + 63) / 64 * 64;
    p.ok = N >= 1024 && p.Dp <= 256 && LM <= 65535 && N < (1ll << 47);
    if (!p.ok) return p;
    p.ntiles = (int)((N + TC_M - 1) / TC_M);
    p.grid = std::min(p.ntiles, num_sms);
    p.ok = false;
    // as few column blocks as fit shared memory with one or two X stages (two
    // unless that takes more blocks: every block reads X again)
    for (int blocks = (LM + 255) / 256; blocks <= (LM + 15) / 16 && !p.ok; ++blocks) {
        p.blk = ((LM + blocks - 1) / blocks + 15) / 16 * 16;
        p.LMp = (LM + p.blk - 1) / p.blk * p.blk;
        p.b_bytes = (uint32_t)p.blk * p.Dp * 2;
        p.x_bytes = (uint32_t)TC_M * p.Dp * 2;
        // operands, barriers, per-column constants, per-thread masks
        const size_t fixed = 1024 + 2 * (size_t)p.b_bytes + 128 + 20 * (size_t)p.blk + 8 * 4 * TC_EPI_WARPS * 32;
        for (int need_lo = 0; need_lo < 2; ++need_lo) {
            const size_t st = (size_t)p.x_bytes * (need_lo ? 2 : 1);
            int stages = 2;
            while (stages > 0 && fixed + stages * st > (size_t)max_smem) --stages;
            p.stages[need_lo] = stages;
            p.smem[need_lo] = fixed + stages * st;
        }
        p.ok = p.stages[1] >= 1;
    }
    return p;
}

cudaError_t launch_project_sample(const float* X, int64_t N, int D, int ns, const float* A, int LM, float slope,
                                  float* xs, float* anorm, ProjectState* ps, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(ps, 0, sizeof(ProjectState), st);
    if (e != cudaSuccess) return e;
    k_project_sample<<<(unsigned)((ns + LM + 7) / 8), 256, 0, st>>>(X, N, D, ns, A, LM, slope, xs, anorm, ps);
    k_project_scales<<<1, 1, 0, st>>>(ps);
    return cudaGetLastError();
}

cudaError_t launch_split_a(const float* A, int LM, int LMp, int D, int Dp, float kappa, float slope, void* ah, void* al, float* anorm,
                           const ProjectState* ps, cudaStream_t st) {
    k_split_a<<<(unsigned)((LMp + 7) / 8), 256, 0, st>>>(A, LM, LMp, D, Dp, kappa, slope, static_cast<__half*>(ah),
                                                        static_cast<__half*>(al), anorm, ps);
    return cudaGetLastError();
}

cudaError_t launch_split_rows(const float* X, int64_t N, int D, int Dp, float kappa, float slope, void* xh, void* xl, float* xnorm,
                              ProjectState* ps, bool rescale, cudaStream_t st) {
    if (rescale) k_project_scales<<<1, 1, 0, st>>>(ps);
    const int blocks = (int)std::min<int64_t>((N * 32 + 255) / 256, 152 * 16);
    k_split_rows<<<blocks, 256, 0, st>>>(X, N, D, Dp, kappa, slope, static_cast<__half*>(xh), static_cast<__half*>(xl), xnorm,
                                        ps);
    return cudaGetLastError();
}

cudaError_t launch_project_tc(const TcPlan& p, int need_lo, int64_t N, int D, int LM, const void* xh, const void* xl,
                              const void* ah, const void* al, const float* b, const float* anorm, const float* xnorm,
                              const ProjectState* ps, float W, float kappa, int32_t* codes, int32_t* pmin, int32_t* pmax,
                              unsigned long long* relist, unsigned long long relist_cap, unsigned int* relist_cnt,
                              int* err, cudaStream_t st) {
    CUtensorMap mxh, mxl, mah, mal;
    if (!make_map(&mxh, xh, p.Dp, N, TC_M) || !make_map(&mxl, need_lo ? xl : xh, p.Dp, N, TC_M) ||
        !make_map(&mah, ah, p.Dp, p.LMp, p.blk) || !make_map(&mal, al, p.Dp, p.LMp, p.blk))
        return cudaErrorNotSupported;
    const int smem = (int)p.smem[need_lo];
    static std::atomic<size_t> opted{0};
    cudaError_t e = opt_in_smem(k_project_tc<false>, p.smem[need_lo], opted);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(relist_cnt, 0, sizeof(unsigned int) * (size_t)p.grid, st);
    if (e != cudaSuccess) return e;
    for (int col0 = 0; col0 < LM; col0 += p.blk) {
        TcArgs a;
        a.N = N;
        a.D = D;
        a.Dp = p.Dp;
        a.LM = std::min(p.blk, LM - col0);
        a.LMp = p.blk;
        a.ntiles = p.ntiles;
        a.need_lo = need_lo;
        a.stages = p.stages[need_lo];
        a.tmem_cols = 32;
        while (a.tmem_cols < 2 * p.blk) a.tmem_cols <<= 1;
        a.W = W;
        a.kappa = kappa;
        a.b = b;
        a.anorm = anorm;
        a.xnorm = xnorm;
        a.ps = ps;
        a.codes = codes;
        a.pmin = pmin;
        a.pmax = pmax;
        a.relist = relist;
        a.relist_cap = relist_cap;
        a.relist_cnt = relist_cnt;
        a.err = err;
        a.b_bytes = p.b_bytes;
        a.x_bytes = p.x_bytes;
        a.col0 = col0;
        a.LMtot = LM;
        a.stage_bytes = 0;
        a.a_chunk = 0;
        k_project_tc<false><<<p.grid, TC_THREADS, smem, st>>>(mxh, mxl, mah, mal, a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

TcStreamPlan tc_plan_stream(int64_t N, int D, int LM, int num_sms, int max_smem) {
    TcStreamPlan p{};
    p.Dp = (D + 63) / 64 * 64;
    p.LMp = (LM + 15) / 16 * 16;
    p.ok = N >= 1024 && p.Dp <= 16384 && LM <= 65535 && N < (1ll << 47);
    if (!p.ok) return p;
    p.ntiles = (int)((N + TC_M - 1) / TC_M);
    p.grid = std::min(p.ntiles, num_sms);
    p.ok = false;
    for (int need_lo = 0; need_lo < 2; ++need_lo) {
        // widest column block whose two-stage (or one-stage) ring fits
        for (int blk = 256; blk >= 16; blk -= 16) {
            const size_t stage = 16384u * (need_lo ? 2u : 1u) + 2u * (size_t)blk * 128u;
            const size_t tail = 128 + 20 * (size_t)blk + 8 * 4 * TC_EPI_WARPS * 32;
            int stages = 2;
            while (stages > 0 && 1024 + stages * stage + tail > (size_t)max_smem) --stages;
            if (stages == 0) continue;
            p.blk[need_lo] = std::min(blk, p.LMp);
            p.stages[need_lo] = stages;
            p.smem[need_lo] = 1024 + stages * (16384u * (need_lo ? 2u : 1u) + 2u * (size_t)p.blk[need_lo] * 128u) +
                              128 + 20 * (size_t)p.blk[need_lo] + 8 * 4 * TC_EPI_WARPS * 32;
            break;
        }
    }
    p.ok = p.stages[1] >= 1 && p.stages[0] >= 1;
    return p;
}

cudaError_t launch_project_tc_stream(const TcStreamPlan& p, int need_lo, int64_t N, int D, int LM, const void* xh,
                                     const void* xl, const void* ah, const void* al, const float* b,
                                     const float* anorm, const float* xnorm, const ProjectState* ps, float W, float kappa,
                                     int32_t* codes, int32_t* pmin, int32_t* pmax, unsigned long long* relist,
                                     unsigned long long relist_cap, unsigned int* relist_cnt, int* err,
                                     cudaStream_t st) {
    const int blk = p.blk[need_lo];
    CUtensorMap mxh, mxl;
    if (!make_map(&mxh, xh, p.Dp, N, TC_M) || !make_map(&mxl, need_lo ? xl : xh, p.Dp, N, TC_M)) return cudaErrorNotSupported;
    const int smem = (int)p.smem[need_lo];
    static std::atomic<size_t> opted{0};
    cudaError_t e = opt_in_smem(k_project_tc<true>, p.smem[need_lo], opted);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(relist_cnt, 0, sizeof(unsigned int) * (size_t)p.grid, st);
    if (e != cudaSuccess) return e;
    for (int col0 = 0; col0 < LM; col0 += blk) {
        const int lmc = std::min(blk, LM - col0);      // columns of this launch
        const int lmp = (lmc + 15) / 16 * 16;           // padded to the MMA's N granularity
        CUtensorMap mah, mal;
        if (!make_map(&mah, ah, p.Dp, (uint64_t)p.LMp, (uint32_t)lmp) ||
            !make_map(&mal, al, p.Dp, (uint64_t)p.LMp, (uint32_t)lmp))
            return cudaErrorNotSupported;
        TcArgs a;
        a.N = N;
        a.D = D;
        a.Dp = p.Dp;
        a.LM = lmc;
        a.LMp = lmp;
        a.ntiles = p.ntiles;
        a.need_lo = need_lo;
        a.stages = p.stages[need_lo];
        int tc = 32;
        while (tc < 2 * lmp) tc <<= 1;
        a.tmem_cols = tc;
        a.W = W;
        a.kappa = kappa;
        a.b = b;
        a.anorm = anorm;
        a.xnorm = xnorm;
        a.codes = codes;
        a.pmin = pmin;
        a.pmax = pmax;
        a.relist = relist;
        a.relist_cap = relist_cap;
        a.relist_cnt = relist_cnt;
        a.ps = ps;
        a.err = err;
        a.b_bytes = 0;
        a.x_bytes = 16384u;
        a.col0 = col0;
        a.LMtot = LM;
        a.a_chunk = (uint32_t)lmp * 128u;
        a.stage_bytes = 16384u * (need_lo ? 2u : 1u) + 2u * a.a_chunk;
        k_project_tc<true><<<p.grid, TC_THREADS, smem, st>>>(mxh, mxl, mah, mal, a);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_tc_recompute(const float* X, int64_t N, int D, int LM, const float* A, const float* b, float W,
                                const unsigned long long* list, unsigned long long cap, const unsigned int* cnt,
                                int regions, int32_t* codes, int32_t* cmin, int32_t* cmax, int* err, cudaStream_t st) {
    // rows of X through shared memory where 16-byte loads apply; A beside them
    // where both fit
    const int stage_x = (D & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const size_t xs = stage_x ? sizeof(float) * (size_t)RT * RP : 0;
    const size_t as = sizeof(float) * (size_t)LM * ((D & 3) == 0 ? D + 4 : D + 1);
    const int stage_a = xs + as <= 215 * 1024;
    const size_t smem = xs + (stage_a ? as : 0);
    static std::atomic<size_t> opted{0};
    cudaError_t e = opt_in_smem(k_tc_recompute, smem, opted);
    if (e != cudaSuccess) return e;
    k_tc_recompute<<<regions, RT, smem, st>>>(X, N, D, A, b, W, list, cap, cnt, regions, LM, stage_a, stage_x, codes, cmin,
                                             cmax, err);
    return cudaGetLastError();
}

}  // namespace culsh
