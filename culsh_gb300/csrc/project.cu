// K1: projection of points onto all L*M stacked LSH columns with the
// bucket-code epilogue fused in.
//
// Replaces cuLSH_Indexing.cu:27-66 (cublasSgemm + kernel_subtractVectorFromMatrixRows
// + kernel_divideMatrixWithScalar) and cuLSH_Kernels.cu:91-101 (kernel_floorMatrix),
// which the reference runs once per table with a full dataset upload each time.
// Here one launch covers every table: C[n][c] = sum_d X[n][d] * A[c][d] over
// c = l*M + m, then v = fl(fl(C) - b) / W and code = floor(v).
//
// Arithmetic is the canonical FP32 order: each output is one fused
// multiply-add chain over d = 0..D-1 in ascending order (register-tiled, the
// tiling never reorders a chain), so codes are bit-exact against the CPU
// oracle. The FP32 FMA pipe bounds this kernel (2*N*D*L*M flops).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "culsh_internal.cuh"

namespace culsh {
namespace {

constexpr int NT = 256;   // threads: 16 (points) x 16 (columns), each PT x CT outputs

// Block tile BN = 16*PT points x BC = 16*CT columns, BK dimensions per
// shared-memory stage. Index builds use PT = 8, CT = 4, BK = 16; query batches
// take one of five tilings the search tuner picks (PT x CT = 4x8 by default,
// 2x8, 8x4, 4x4, 2x4: fewer shared-memory loads per FMA against more blocks
// in flight), and 2x12 (all of L*M <= 192 columns in one block) when the
// queries are read straight from host memory and copied to the device on
// the way (xcopy).
//
// Thread (tx, ty) owns points 32*(i/2) + 2*tx + (i%2), i < PT, so that a
// half-warp's float2 reads of the X tile cover 128 contiguous bytes (no bank
// conflicts), and columns ty*CT .. ty*CT+CT-1. The projection matrix is read
// transposed (AT[d][c], rows of lmp >= LM floats, columns past LM zero) with
// coalesced float4 loads. The next stage's tiles are loaded into registers
// while the current one is multiplied.
template <bool kCodes, int PT, int CT, int BK, bool kCopy = false>
__global__ void __launch_bounds__(NT, kCopy ? 2 : 0) k_project(const float* __restrict__ X, int64_t n_pts, int D,
                                                const float* __restrict__ AT, int lmp, const float* __restrict__ b,
                                                int LM, float W, int32_t* __restrict__ codes,
                                                float* __restrict__ vals, int32_t* __restrict__ pmin,
                                                int32_t* __restrict__ pmax, int* __restrict__ err,
                                                ZeroWords zw, float* __restrict__ xcopy) {
    constexpr int BN = 16 * PT;
    constexpr int BC = 16 * CT;
    constexpr int XP = BN + 2;   // padded X row: the transposing stores conflict at most 4 ways
    constexpr int XS = BN * BK / NT;        // X floats per thread per stage
    constexpr int AV = BC * BK / 4 / NT;    // AT float4 per thread per stage
    static_assert(PT % 2 == 0 && XS % 4 == 0 && AV >= 1 && BC * BK == AV * 4 * NT, "tile shape");
    static_assert(BK % 16 == 0, "As must start 16-byte aligned");
    constexpr int kTileBytes = BK * (XP + BC) * 4;
    constexpr int kStageBytes = BC * (BN + 1) * 4;
    // The epilogue's staging reuses the tiles (the main loop ends on a barrier).
    __shared__ __align__(16) unsigned char smem[kTileBytes > kStageBytes ? kTileBytes : kStageBytes];
    float (*Xs)[XP] = reinterpret_cast<float (*)[XP]>(smem);
    float (*As)[BC] = reinterpret_cast<float (*)[BC]>(smem + BK * XP * 4);
    uint32_t (*Cs)[BN + 1] = reinterpret_cast<uint32_t (*)[BN + 1]>(smem);

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    zw.clear(tid);
    const int64_t n0 = (int64_t)blockIdx.x * BN;
    const int c0 = blockIdx.y * BC;
    const bool vec = (D & 3) == 0;

    float xr[XS];
    float4 ar[AV];
    // Global -> registers. Vector path: BK/4 consecutive threads read one
    // point's BK dimensions; scalar path (D % 4 != 0): BK threads do. Zero
    // fill past D adds +-0 to a chain, which leaves it unchanged.
    auto gload = [&](int d0) {
        if (vec) {
#pragma unroll
            for (int r = 0; r < XS / 4; ++r) {
                const int f = tid + NT * r, dq = f % (BK / 4), p = f / (BK / 4);
                const int64_t gn = n0 + p;
                const int gd = d0 + dq * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (gn < n_pts && gd < D) {
                    v = __ldg(reinterpret_cast<const float4*>(X + gn * D + gd));
                    if constexpr (kCopy) *reinterpret_cast<float4*>(xcopy + gn * D + gd) = v;
                }
                xr[4 * r + 0] = v.x;
                xr[4 * r + 1] = v.y;
                xr[4 * r + 2] = v.z;
                xr[4 * r + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int r = 0; r < XS; ++r) {
                const int f = tid + NT * r, dd = f % BK, p = f / BK;
                const int64_t gn = n0 + p;
                const int gd = d0 + dd;
                xr[r] = (gn < n_pts && gd < D) ? __ldg(X + gn * D + gd) : 0.0f;
                if constexpr (kCopy) {
                    if (gn < n_pts && gd < D) xcopy[gn * D + gd] = xr[r];
                }
            }
        }
#pragma unroll
        for (int r = 0; r < AV; ++r) {
            const int f = tid + NT * r, cq = f % (BC / 4), dd = f / (BC / 4);
            const int gc = c0 + cq * 4, gd = d0 + dd;
            ar[r] = (gc < lmp && gd < D) ? __ldg(reinterpret_cast<const float4*>(AT + (int64_t)gd * lmp + gc))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto sstore = [&]() {
        if (vec) {
#pragma unroll
            for (int r = 0; r < XS / 4; ++r) {
                const int f = tid + NT * r, dq = f % (BK / 4), p = f / (BK / 4);
#pragma unroll
                for (int e = 0; e < 4; ++e) Xs[dq * 4 + e][p] = xr[4 * r + e];
            }
        } else {
#pragma unroll
            for (int r = 0; r < XS; ++r) {
                const int f = tid + NT * r, dd = f % BK, p = f / BK;
                Xs[dd][p] = xr[r];
            }
        }
#pragma unroll
        for (int r = 0; r < AV; ++r) {
            const int f = tid + NT * r, cq = f % (BC / 4), dd = f / (BC / 4);
            *reinterpret_cast<float4*>(&As[dd][cq * 4]) = ar[r];
        }
    };

    float acc[PT][CT];
#pragma unroll
    for (int i = 0; i < PT; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) acc[i][j] = 0.0f;

    gload(0);
    for (int d0 = 0; d0 < D; d0 += BK) {
        sstore();
        __syncthreads();
        if (d0 + BK < D) gload(d0 + BK);
#pragma unroll 8
        for (int k = 0; k < BK; ++k) {
            float xv[PT];
#pragma unroll
            for (int i = 0; i < PT; i += 2) {
                const float2 x2 = *reinterpret_cast<const float2*>(&Xs[k][16 * i + 2 * tx]);
                xv[i] = x2.x;
                xv[i + 1] = x2.y;
            }
            float aw[CT];
#pragma unroll
            for (int j = 0; j < CT; j += 4) {
                const float4 av = *reinterpret_cast<const float4*>(&As[k][ty * CT + j]);
                aw[j] = av.x;
                aw[j + 1] = av.y;
                aw[j + 2] = av.z;
                aw[j + 3] = av.w;
            }
#pragma unroll
            for (int i = 0; i < PT; ++i)
#pragma unroll
                for (int j = 0; j < CT; ++j) acc[i][j] = __fmaf_rn(xv[i], aw[j], acc[i][j]);
        }
        __syncthreads();
    }

    // Epilogue: -b, /W (IEEE divide), floor; stage through shared memory for
    // coalesced column-major stores.
    int bad = 0;
#pragma unroll
    for (int j = 0; j < CT; ++j) {
        const int c = c0 + ty * CT + j;
        const float bc = (c < LM) ? __ldg(b + c) : 0.0f;
        int32_t lo = INT_MAX, hi = INT_MIN;
#pragma unroll
        for (int i = 0; i < PT; ++i) {
            const int pi = 16 * (i & ~1) + 2 * tx + (i & 1);
            const float v = __fdiv_rn(__fsub_rn(acc[i][j], bc), W);
            uint32_t bits;
            if (kCodes) {
                const float f = floorf(v);
                int32_t code = 0;
                if (!(fabsf(f) <= FLT_MAX)) {
                    bad |= kErrNonFinite;
                } else if (!(f >= -2147483648.0f && f < 2147483648.0f)) {
                    bad |= kErrCodeRange;
                } else {
                    code = (int32_t)f;
                }
                if (n0 + pi < n_pts && c < LM) {
                    lo = min(lo, code);
                    hi = max(hi, code);
                }
                bits = (uint32_t)code;
            } else {
                bits = __float_as_uint(v);
            }
            Cs[ty * CT + j][pi] = bits;
        }
        if (kCodes) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if (tx == 0 && c < LM) {
                pmin[(int64_t)blockIdx.x * LM + c] = lo;
                pmax[(int64_t)blockIdx.x * LM + c] = hi;
            }
        }
    }
    if (kCodes && bad) atomicOr(err, bad);
    __syncthreads();
    constexpr int RPI = NT / BN;   // rows stored per iteration
    const int p = tid % BN;
#pragma unroll 4
    for (int r = 0; r < BC / RPI; ++r) {
        const int row = r * RPI + tid / BN;
        const int c = c0 + row;
        if (c < LM && n0 + p < n_pts) {
            const int64_t o = (int64_t)c * n_pts + n0 + p;
            if (kCodes) codes[o] = (int32_t)Cs[row][p];
            else vals[o] = __uint_as_float(Cs[row][p]);
        }
    }
}

// Few queries: one column per thread, P rows per block of 64 columns, the rows
// staged whole and a column's next 16 values loaded while 16 are multiplied.
// Bound by the latency of those loads; the tilings above, made for ten thousand
// queries, leave most SMs without a block and wait for one stage of 32 dimensions
// after another (128 dimensions: one query on 64 columns 14 us, now 5; 1,000 on
// 64 17, now 11; 256 on 192 15, now 10).
// Same chains, same parameters as k_project (vals only).
constexpr int FC = 64;     // columns (threads)
constexpr int FD = 256;    // dimensions at most
template <int P>
__global__ void __launch_bounds__(FC) k_project_few(const float* __restrict__ X, int64_t n_pts, int D,
                                                    const float* __restrict__ AT, int lmp, const float* __restrict__ b,
                                                    int LM, float W, int32_t*, float* __restrict__ vals, int32_t*,
                                                    int32_t*, int*, ZeroWords zw, float* __restrict__ xcopy) {
    __shared__ __align__(16) float xs[P][FD];
    const int tid = threadIdx.x, c = blockIdx.y * FC + tid;
    zw.clear(tid);
    const int64_t n0 = (int64_t)blockIdx.x * P;
    const int rows = (int)min((int64_t)P, n_pts - n0);
    const bool vec = (D & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const bool copy = xcopy && blockIdx.y == 0;
    const float* at = AT + min(c, lmp - 1);
    float acc[P];
#pragma unroll
    for (int p = 0; p < P; ++p) acc[p] = 0.0f;
    const int dp = (D + 15) & ~15;
    float cur[16], nxt[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) cur[i] = i < D ? __ldg(at + (int64_t)i * lmp) : 0.0f;
    // dimensions past D are zeros: they leave a chain unchanged
    if (vec) {
#pragma unroll 4
        for (int f = tid; f < P * (dp / 4); f += FC) {
            const int p = f / (dp / 4), d = f % (dp / 4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p < rows && d < D) {
                v = __ldg(reinterpret_cast<const float4*>(X + (n0 + p) * D + d));
                if (copy) *reinterpret_cast<float4*>(xcopy + (n0 + p) * D + d) = v;
            }
            *reinterpret_cast<float4*>(&xs[p][d]) = v;
        }
    } else {
#pragma unroll 4
        for (int f = tid; f < P * dp; f += FC) {
            const int p = f / dp, d = f % dp;
            const float v = p < rows && d < D ? __ldg(X + (n0 + p) * D + d) : 0.0f;
            if (copy && p < rows && d < D) xcopy[(n0 + p) * D + d] = v;
            xs[p][d] = v;
        }
    }
    __syncthreads();
    for (int d = 0; d < dp; d += 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) nxt[i] = d + 16 + i < D ? __ldg(at + (int64_t)(d + 16 + i) * lmp) : 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i += 4)
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const float4 x = *reinterpret_cast<const float4*>(&xs[p][d + i]);
                acc[p] = __fmaf_rn(x.x, cur[i], acc[p]);
                acc[p] = __fmaf_rn(x.y, cur[i + 1], acc[p]);
                acc[p] = __fmaf_rn(x.z, cur[i + 2], acc[p]);
                acc[p] = __fmaf_rn(x.w, cur[i + 3], acc[p]);
            }
#pragma unroll
        for (int i = 0; i < 16; ++i) cur[i] = nxt[i];
    }
    if (c >= LM) return;
    const float bc = __ldg(b + c);
    float* out = vals + (int64_t)c * n_pts + n0;
#pragma unroll
    for (int p = 0; p < P; ++p)
        if (p < rows) out[p] = __fdiv_rn(__fsub_rn(acc[p], bc), W);
}

// Rows per block of the few-queries form, 0 where the tilings take over: when
// they have more than 64 blocks, or more than 256 dimensions (all blocks read
// the same rows of AT at the same time: 256 queries of 960 dimensions on 512
// columns take 58 us in both, 1,000 take 68 and 58).
int few_rows(int64_t n_pts, int D, int LM) {
    if (D > 256 || ((n_pts + 63) / 64) * ((LM + 127) / 128) > 64) return 0;
    return n_pts <= 64 ? 2 : 8;
}
typedef void (*FewKernel)(const float*, int64_t, int, const float*, int, const float*, int, float, int32_t*, float*,
                          int32_t*, int32_t*, int*, ZeroWords, float*);
FewKernel few_kernel(int rows) { return rows == 2 ? k_project_few<2> : k_project_few<8>; }

// Wide tiling of the index build's projection: 128 points x 128 columns per
// block, 8 x 8 outputs per thread, 16 dimensions per stage, two stages in shared
// memory (the next one's loads are in registers while this one is multiplied).
// Same chains as k_project: each output is one FMA chain in ascending d, held
// in packed pairs of columns (two FMAs per instruction). Per dimension a thread
// reads 16 floats for 64 FMAs; the 8 x 4 tiling reads 12 for 32 and left the
// FMA pipe half idle on shared-memory and issue slots (1M x 960 points, 512
// columns: 23.3 ms, 42 of the pipe's 80 TFLOP/s; this tiling 16.9 ms).
constexpr int WB = 128;        // points and columns of a block
constexpr int WK = 16;         // dimensions per stage
constexpr int WP = WB + 4;     // padded row of a stage (16-byte rows)

__global__ void __launch_bounds__(NT, 2) k_project_wide(const float* __restrict__ X, int64_t n_pts, int D,
                                                        const float* __restrict__ AT, int lmp,
                                                        const float* __restrict__ b, int LM, float W,
                                                        int32_t* __restrict__ codes, int32_t* __restrict__ pmin,
                                                        int32_t* __restrict__ pmax, int* __restrict__ err) {
    __shared__ __align__(16) float Xs[2][WK][WP];
    __shared__ __align__(16) float As[2][WK][WP];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t n0 = (int64_t)blockIdx.x * WB;
    const int c0 = blockIdx.y * WB;
    const bool vec = (D & 3) == 0;
    // X: thread reads float4 number tid % 4 of points tid / 4 and tid / 4 + 64;
    // AT: float4 number tid % 32 of dimensions tid / 32 and tid / 32 + 8
    const int xd = (tid & 3) * 4, xp = tid >> 2, ac = (tid & 31) * 4, ad = tid >> 5;
    float4 xr[2], ar[2];
    auto gload = [&](int d0) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t gn = n0 + xp + 64 * r;
            const int gd = d0 + xd;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);   // adds +-0 to a chain past D
            if (gn < n_pts) {
                const float* row = X + gn * D;
                if (vec) {
                    if (gd < D) v = __ldg(reinterpret_cast<const float4*>(row + gd));
                } else {
                    if (gd < D) v.x = __ldg(row + gd);
                    if (gd + 1 < D) v.y = __ldg(row + gd + 1);
                    if (gd + 2 < D) v.z = __ldg(row + gd + 2);
                    if (gd + 3 < D) v.w = __ldg(row + gd + 3);
                }
            }
            xr[r] = v;
            const int da = d0 + ad + 8 * r;
            ar[r] = c0 + ac < lmp && da < D ? __ldg(reinterpret_cast<const float4*>(AT + (int64_t)da * lmp + c0 + ac))
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto sstore = [&](int st) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            Xs[st][xd + 0][xp + 64 * r] = xr[r].x;
            Xs[st][xd + 1][xp + 64 * r] = xr[r].y;
            Xs[st][xd + 2][xp + 64 * r] = xr[r].z;
            Xs[st][xd + 3][xp + 64 * r] = xr[r].w;
            *reinterpret_cast<float4*>(&As[st][ad + 8 * r][ac]) = ar[r];
        }
    };
    // outputs: points 4 tx + {0..3} and 64 + 4 tx + {0..3}, columns 4 ty + {0..3}
    // and 64 + 4 ty + {0..3} in pairs
    float2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
    gload(0);
    sstore(0);
    __syncthreads();
    int st = 0;
    for (int d0 = 0; d0 < D; d0 += WK, st ^= 1) {
        if (d0 + WK < D) gload(d0 + WK);
#pragma unroll
        for (int k = 0; k < WK; ++k) {
            const float4 x0 = *reinterpret_cast<const float4*>(&Xs[st][k][4 * tx]);
            const float4 x1 = *reinterpret_cast<const float4*>(&Xs[st][k][64 + 4 * tx]);
            const float4 a0 = *reinterpret_cast<const float4*>(&As[st][k][4 * ty]);
            const float4 a1 = *reinterpret_cast<const float4*>(&As[st][k][64 + 4 * ty]);
            const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            const float2 av[4] = {make_float2(a0.x, a0.y), make_float2(a0.z, a0.w), make_float2(a1.x, a1.y),
                                  make_float2(a1.z, a1.w)};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(xv[i], xv[i]), av[j], acc[i][j]);
        }
        if (d0 + WK < D) sstore(st ^ 1);   // the other stage: last read before the previous barrier
        __syncthreads();
    }

    // -b, /W (IEEE divide), floor; four consecutive points of a column per store
    const bool st4 = (n_pts & 3) == 0;
    int bad = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = c0 + (j >> 2) * 64 + ty * 4 + (j & 3);
        const float bc = c < LM ? __ldg(b + c) : 0.0f;
        int32_t lo = INT_MAX, hi = INT_MIN;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int32_t code[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a2 = acc[h * 4 + i][j >> 1];
                const float f = floorf(__fdiv_rn(__fsub_rn((j & 1) ? a2.y : a2.x, bc), W));
                code[i] = 0;
                if (!(fabsf(f) <= FLT_MAX)) bad |= kErrNonFinite;
                else if (!(f >= -2147483648.0f && f < 2147483648.0f)) bad |= kErrCodeRange;
                else code[i] = (int32_t)f;
                if (n0 + h * 64 + 4 * tx + i < n_pts) {
                    lo = min(lo, code[i]);
                    hi = max(hi, code[i]);
                }
            }
            const int64_t n = n0 + h * 64 + 4 * tx;
            if (c < LM && n < n_pts) {
                int32_t* o = codes + (int64_t)c * n_pts + n;
                if (st4) {
                    *reinterpret_cast<int4*>(o) = make_int4(code[0], code[1], code[2], code[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (n + i < n_pts) o[i] = code[i];
                }
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (tx == 0 && c < LM) {
            pmin[(int64_t)blockIdx.x * LM + c] = lo;
            pmax[(int64_t)blockIdx.x * LM + c] = hi;
        }
    }
    if (bad) atomicOr(err, bad);
}

__global__ void k_minmax_reduce(const int32_t* __restrict__ pmin, const int32_t* __restrict__ pmax, int nparts, int LM,
                                int32_t* __restrict__ cmin, int32_t* __restrict__ cmax) {
    const int c = blockIdx.x;
    int32_t lo = INT_MAX, hi = INT_MIN;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        lo = min(lo, pmin[(int64_t)i * LM + c]);
        hi = max(hi, pmax[(int64_t)i * LM + c]);
    }
    __shared__ int32_t slo[32], shi[32];
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        slo[w] = lo;
        shi[w] = hi;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        lo = lane < nw ? slo[lane] : INT_MAX;
        hi = lane < nw ? shi[lane] : INT_MIN;
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            cmin[c] = lo;
            cmax[c] = hi;
        }
    }
}

}  // namespace

// Index builds (codes) use 128-point tiles; query batches (values) use
// 64-point tiles so that ten thousand queries still fill every SM.
int project_grid_x(int64_t n_pts) { return (int)((n_pts + 127) / 128); }

cudaError_t launch_project_fp32(const float* X, int64_t n_pts, int D, const float* AT, int lmp, const float* b,
                                int LM, float W, int32_t* codes, float* vals, int32_t* pmin, int32_t* pmax, int* err,
                                cudaStream_t st, int tile, ZeroWords zw, float* xcopy) {
    if (n_pts <= 0) return cudaSuccess;
    if (lmp < LM || (lmp & 3) || ((uintptr_t)AT & 15)) return cudaErrorInvalidValue;
    // xcopy (the rows also written to device memory as they are read): one
    // column block, so that every row is read exactly once
    if (xcopy && (codes || tile != 5 || LM > 192)) return cudaErrorInvalidValue;
    const int few = !codes && (tile == 0 || tile == 5) ? few_rows(n_pts, D, LM) : 0;
    if (few) {
        few_kernel(few)<<<dim3((unsigned)((n_pts + few - 1) / few), (LM + FC - 1) / FC), FC, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, xcopy);
    } else if (codes && LM > 64) {
        // one column block of 64 (LM <= 64) would leave half of the wide tile idle
        k_project_wide<<<dim3(project_grid_x(n_pts), (LM + WB - 1) / WB), NT, 0, st>>>(X, n_pts, D, AT, lmp, b, LM, W,
                                                                                     codes, pmin, pmax, err);
    } else if (codes) {
        k_project<true, 8, 4, 16><<<dim3(project_grid_x(n_pts), (LM + 63) / 64), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, codes, nullptr, pmin, pmax, err, zw, nullptr);
    } else if (tile == 1) {
        k_project<false, 2, 8, 64><<<dim3((unsigned)((n_pts + 31) / 32), (LM + 127) / 128), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, nullptr);
    } else if (tile == 2) {
        k_project<false, 8, 4, 32><<<dim3((unsigned)((n_pts + 127) / 128), (LM + 63) / 64), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, nullptr);
    } else if (tile == 3) {
        k_project<false, 4, 4, 32><<<dim3((unsigned)((n_pts + 63) / 64), (LM + 63) / 64), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, nullptr);
    } else if (tile == 4) {
        k_project<false, 2, 4, 32><<<dim3((unsigned)((n_pts + 31) / 32), (LM + 63) / 64), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, nullptr);
    } else if (tile == 5) {
        if (!xcopy) return cudaErrorInvalidValue;   // tiling 5 serves the copying form only
        k_project<false, 2, 12, 32, true><<<dim3((unsigned)((n_pts + 31) / 32), (LM + 191) / 192), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, xcopy);
    } else {
        k_project<false, 4, 8, 32><<<dim3((unsigned)((n_pts + 63) / 64), (LM + 127) / 128), NT, 0, st>>>(
            X, n_pts, D, AT, lmp, b, LM, W, nullptr, vals, nullptr, nullptr, err, zw, nullptr);
    }
    return cudaGetLastError();
}

template <typename F>
struct arity;
template <typename R, typename... A>
struct arity<R(A...)> {
    static constexpr int value = sizeof...(A);
};
static_assert(arity<decltype(k_project<false, 2, 12, 32, true>)>::value == kProjectArgs, "projection parameters");

static_assert(arity<std::remove_pointer_t<FewKernel>>::value == kProjectArgs, "projection parameters");

const void* project_copy_kernel(int64_t n_pts, int D, int LM) {
    const int few = few_rows(n_pts, D, LM);
    if (few) return reinterpret_cast<const void*>(few_kernel(few));
    return reinterpret_cast<const void*>(&k_project<false, 2, 12, 32, true>);
}

cudaError_t launch_minmax_reduce(const int32_t* pmin, const int32_t* pmax, int nparts, int LM, int32_t* cmin,
                                 int32_t* cmax, cudaStream_t st) {
    k_minmax_reduce<<<LM, 256, 0, st>>>(pmin, pmax, nparts, LM, cmin, cmax);
    return cudaGetLastError();
}

// Copies n floats from src (16-byte aligned; host memory the device can read,
// or device memory) to dst with 16-byte loads: one pass over the source. Each
// thread issues kCopyVec independent loads before its stores, so that reads
// over the host link (microseconds of latency) overlap.
constexpr int kCopyVec = 8;

__global__ void __launch_bounds__(256) k_copy_f32(const float* __restrict__ src, float* __restrict__ dst, int64_t n) {
    const int64_t n4 = n >> 2;
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    const int64_t base = (int64_t)blockIdx.x * (256 * kCopyVec) + threadIdx.x;
    float4 v[kCopyVec];
#pragma unroll
    for (int k = 0; k < kCopyVec; ++k) {
        const int64_t i = base + (int64_t)k * 256;
        if (i < n4) v[k] = s4[i];
    }
#pragma unroll
    for (int k = 0; k < kCopyVec; ++k) {
        const int64_t i = base + (int64_t)k * 256;
        if (i < n4) d4[i] = v[k];
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) dst[(n4 << 2) + threadIdx.x] = src[(n4 << 2) + threadIdx.x];
}

cudaError_t launch_copy_f32(const float* src, float* dst, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (((uintptr_t)src & 15) || ((uintptr_t)dst & 15)) return cudaErrorInvalidValue;
    const int64_t blocks = ((n >> 2) + 256 * kCopyVec - 1) / (256 * kCopyVec);
    k_copy_f32<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, st>>>(src, dst, n);
    return cudaGetLastError();
}

}  // namespace culsh
