// K2 + K3: bucketing of the projected codes.
//
// Replaces cuLSH_Indexing.cu:71-93 (radixSortRows_1matrix: M gather + stable
// sort passes over float columns, per table) and cuLSH_Indexing.cu:98-169
// (calculateBuckets / copyMatrixRows: boundary flags, counts, unique codes).
//
// Each point's code row of table l is packed into a multi-word key: column m
// becomes a field of bit width fbits[l*M+m] (enough for cmax - cmin), column 0
// in the most significant bits, so unsigned key order equals the reference's
// lexicographic order on (c0, c1, ..., c_{M-1}). All L tables are sorted in
// one onesweep LSD radix sort (8-bit digits, decoupled look-back, one launch
// per digit pass over all tables); the sort is stable and starts from id
// order, so ids inside a bucket ascend as in the reference. A run-length pass
// then emits bucket starts, sizes and unique keys, and an open-addressing hash
// over the unique keys serves exact-code lookups at query time.
//
// Every pass streams keys and ids once in and once out (the digit's own
// word is read once; the first pass makes the ids).
#include <algorithm>
#include <climits>

#include "culsh_internal.cuh"

namespace culsh {
namespace {

constexpr int NT = 256;
constexpr int SP_ITEMS = 16;
constexpr int SP_TILE = NT * SP_ITEMS;      // 4096 elements per tile
constexpr int SP_WARPS = NT / 32;
constexpr uint32_t ST_AGG = 1u << 30;       // tile aggregate published
constexpr uint32_t ST_PRE = 2u << 30;       // inclusive prefix published
constexpr uint32_t ST_CNT = (1u << 30) - 1;
constexpr int HIST_CHUNK = 8192;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr int kRunMax = 2048;               // longest run of equal top words ordered in shared memory

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Exclusive scan of one value per thread over a 256-thread block.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t t = lane < SP_WARPS ? ws[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < SP_WARPS) ws[lane] = t;
    }
    __syncthreads();
    const uint32_t pre = w > 0 ? ws[w - 1] : 0;
    if (total) *total = ws[SP_WARPS - 1];
    const uint32_t r = pre + x - v;
    __syncthreads();
    return r;
}

// Keys of one table's points (blockIdx.y), PK_ITEMS per thread. Fields are
// contiguous from column M - 1's offset upwards; a column's bit width and
// offset are the same for every thread, so the words are filled from a 64-bit
// window with uniform control flow (a 128-bit shift per column had cost 44
// instructions per code: 0.38 ms for 1M x 192 codes, now 0.23 ms).
// WIDE: keys of more than 128 bits (KW > 4), assembled word by word.
constexpr int PK_ITEMS = 4;
template <bool WIDE>
__global__ void __launch_bounds__(NT) k_pack_keys(const int32_t* __restrict__ codes, int64_t N, int L, int M, int KW,
                            const int32_t* __restrict__ cmin, const uint8_t* __restrict__ fbits,
                            const uint16_t* __restrict__ foff, uint32_t* __restrict__ keys,
                            uint32_t* __restrict__ vals, uint32_t* __restrict__ low, int lw) {
    const int64_t LN = (int64_t)L * N;
    const int l = blockIdx.y;
    const int64_t n0 = (int64_t)blockIdx.x * (NT * PK_ITEMS) + threadIdx.x;
    const int32_t* cl = codes + (int64_t)l * M * N;
    if constexpr (WIDE) {
        for (int i = 0; i < PK_ITEMS; ++i) {
            const int64_t n = n0 + i * NT;
            if (n >= N) break;
            uint32_t key[kMaxKW] = {};
            for (int m = 0; m < M; ++m) {
                const int c = l * M + m;
                const int bits = __ldg(fbits + c);
                if (bits) key_put(key, __ldg(foff + c), bits, (uint32_t)(cl[(int64_t)m * N + n] - __ldg(cmin + c)));
            }
            for (int w = 0; w < KW; ++w) keys[w * LN + (int64_t)l * N + n] = key[w];
            if (vals) vals[(int64_t)l * N + n] = (uint32_t)n;
        }
    } else {
        uint32_t k[4][PK_ITEMS];
        uint64_t acc[PK_ITEMS];
#pragma unroll
        for (int i = 0; i < PK_ITEMS; ++i) {
            acc[i] = 0;
#pragma unroll
            for (int w = 0; w < 4; ++w) k[w][i] = 0;
        }
        int pos = __ldg(foff + l * M + M - 1), w = 0;   // next bit within the window, word at its bottom
        auto emit = [&]() {   // the window's low word is complete
#pragma unroll
            for (int i = 0; i < PK_ITEMS; ++i) {
                const uint32_t v = (uint32_t)acc[i];
                if (w == 0) k[0][i] = v;
                else if (w == 1) k[1][i] = v;
                else if (w == 2) k[2][i] = v;
                else k[3][i] = v;
                acc[i] >>= 32;
            }
            ++w;
            pos -= 32;
        };
        while (pos >= 32) emit();
        for (int m = M - 1; m >= 0; --m) {
            const int c = l * M + m;
            const int bits = __ldg(fbits + c);
            if (bits == 0) continue;
            const int32_t lo = __ldg(cmin + c);
#pragma unroll
            for (int i = 0; i < PK_ITEMS; ++i) {
                const int64_t n = n0 + i * NT;
                const uint32_t f = n < N ? (uint32_t)(__ldcs(cl + (int64_t)m * N + n) - lo) : 0u;
                acc[i] |= (uint64_t)f << pos;
            }
            pos += bits;
            if (pos >= 32) emit();
        }
        if (pos > 0) emit();
#pragma unroll
        for (int i = 0; i < PK_ITEMS; ++i) {
            const int64_t n = n0 + i * NT, idx = (int64_t)l * N + n;
            if (n >= N) break;
            if (low) {   // top-word-first form: the top word in keys, the lower ones as a row
                keys[idx] = lw == 1 ? k[1][i] : lw == 2 ? k[2][i] : k[3][i];
                if (lw == 1) low[idx] = k[0][i];
                else if (lw == 2) reinterpret_cast<uint2*>(low)[idx] = make_uint2(k[0][i], k[1][i]);
                else reinterpret_cast<uint4*>(low)[idx] = make_uint4(k[0][i], k[1][i], k[2][i], 0u);
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (v < KW) keys[v * LN + idx] = k[v][i];
            }
            if (vals) vals[idx] = (uint32_t)n;
        }
    }
}

__global__ void k_sort_hist(const uint32_t* __restrict__ keys, int64_t N, int L, int passes,
                            uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t sh[];
    for (int i = threadIdx.x; i < passes * 256; i += NT) sh[i] = 0;
    __syncthreads();
    const int l = blockIdx.y;
    const int64_t LN = (int64_t)L * N, seg = (int64_t)l * N;
    const int64_t start = (int64_t)blockIdx.x * HIST_CHUNK;
    const int64_t end = min(N, start + HIST_CHUNK);
    for (int w = 0; w * 4 < passes; ++w) {
        const uint32_t* kw = keys + w * LN + seg;
        const int np = min(4, passes - 4 * w);
        for (int64_t i = start + threadIdx.x; i < end; i += NT) {
            const uint32_t k = kw[i];
            for (int s = 0; s < np; ++s) atomicAdd(&sh[(4 * w + s) * 256 + ((k >> (8 * s)) & 255u)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += NT)
        if (sh[i]) atomicAdd(&hist[(int64_t)l * passes * 256 + i], sh[i]);
}

__global__ void k_sort_digit_base(const uint32_t* __restrict__ hist, uint32_t* __restrict__ base) {
    __shared__ uint32_t ws[SP_WARPS];
    const int64_t o = (int64_t)blockIdx.x * 256 + threadIdx.x;
    base[o] = block_excl_scan(hist[o], ws, nullptr);
}

// Positions of two consecutive items of a warp (digits d0, then d1 of each
// lane) among the warp's elements of the same digit. The lanes of one digit
// find one another through a mask word per digit that each sets its bit in (a
// match instruction per item had taken half of a pass: 0.51 ms for four passes
// over 16M pairs against 0.32; eight ballots 0.43), the highest of them counts
// for all and clears the word. wm: two arrays of 256 zeroed mask words, wh: the
// warp's 256 counters. Two items share the waits.
__device__ __forceinline__ void rank_two(uint32_t* wm, uint32_t* wh, uint32_t d0, uint32_t d1, uint32_t& r0, uint32_t& r1) {
    const int lane = threadIdx.x & 31;
    atomicOr(wm + d0, 1u << lane);
    atomicOr(wm + 256 + d1, 1u << lane);
    __syncwarp();
    const uint32_t p0 = wm[d0], p1 = wm[256 + d1];
    __syncwarp();
    const int l0 = 31 - __clz((int)p0), l1 = 31 - __clz((int)p1);
    uint32_t b0 = 0, b1 = 0;
    if (lane == l0) {
        wm[d0] = 0;
        b0 = atomicAdd(wh + d0, (uint32_t)__popc(p0));
    }
    __syncwarp();   // the second item counts after the first
    if (lane == l1) {
        wm[256 + d1] = 0;
        b1 = atomicAdd(wh + d1, (uint32_t)__popc(p1));
    }
    __syncwarp();
    r0 = __shfl_sync(0xffffffffu, b0, l0) + __popc(p0 & ((1u << lane) - 1u));
    r1 = __shfl_sync(0xffffffffu, b1, l1) + __popc(p1 & ((1u << lane) - 1u));
}

// One LSD digit pass over all tables. Tiles are taken in launch order from a
// global counter, so every tile's predecessors have started before it and the
// look-back wait always ends; it is bounded anyway (kErrSpin).
__global__ void __launch_bounds__(NT, 3) k_sort_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                  uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                  int64_t N, int L, int KW, int tiles, int word, int shift,
                                                  const uint32_t* __restrict__ base, int passes, int pass,
                                                  uint32_t* status, uint32_t* counter, int* err) {
    __shared__ uint32_t whist[SP_WARPS][256];
    __shared__ uint32_t tstart[256];
    __shared__ uint32_t gadd[256];
    __shared__ uint32_t buf[SP_TILE];
    __shared__ uint32_t wtile[SP_TILE];
    __shared__ uint8_t sdig[SP_TILE];
    __shared__ uint32_t ws[SP_WARPS];
    __shared__ uint32_t s_vb;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_vb = atomicAdd(counter, 1u);
    for (int i = tid; i < SP_WARPS * 256; i += NT) (&whist[0][0])[i] = 0;
    for (int i = tid; i < SP_TILE; i += NT) buf[i] = 0;   // mask words of the ranking (SP_TILE >= 512 a warp)
    __syncthreads();
    const uint32_t vb = s_vb;
    const int l = (int)(vb / (uint32_t)tiles), tile = (int)(vb % (uint32_t)tiles);
    const int64_t LN = (int64_t)L * N, seg = (int64_t)l * N;
    const int64_t t0 = (int64_t)tile * SP_TILE;
    const int nvalid = (N - t0 < SP_TILE) ? (int)(N - t0) : SP_TILE;
    const uint32_t* kw = kin + word * LN + seg + t0;

    uint32_t dig[SP_ITEMS], pos[SP_ITEMS];
#pragma unroll
    for (int i = 0; i < SP_ITEMS; ++i) {
        const int e = warp * (32 * SP_ITEMS) + i * 32 + lane;
        const uint32_t w = (e < nvalid) ? kw[e] : 0u;
        wtile[e] = w;   // the digit's key word, kept for its own scatter
        dig[i] = (e < nvalid) ? ((w >> shift) & 255u) : 256u;
    }
    // Stable warp-level ranking: element order inside a warp chunk is
    // (item, lane), which is the element order of the tile. Elements past the
    // end count as the largest digit, after all others.
#pragma unroll
    for (int i = 0; i < SP_ITEMS; i += 2)
        rank_two(buf + warp * 512, whist[warp], min(dig[i], 255u), min(dig[i + 1], 255u), pos[i], pos[i + 1]);
    __syncthreads();
    // Thread tid owns digit tid: per-warp exclusive offsets and tile total.
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < SP_WARPS; ++w) {
        const uint32_t c = whist[w][tid];
        whist[w][tid] = run;
        run += c;
    }
    const uint32_t total = tid == 255 ? run - (uint32_t)(SP_TILE - nvalid) : run;
    tstart[tid] = block_excl_scan(total, ws, nullptr);

    // Decoupled look-back for digit tid.
    uint32_t* my = status + ((int64_t)l * tiles + tile) * 256 + tid;
    uint32_t excl = 0;
    if (tile == 0) {
        st_relaxed(my, ST_PRE | total);
    } else {
        st_relaxed(my, ST_AGG | total);
        int j = tile - 1;
        uint32_t spins = 0;
        while (j >= 0) {
            const uint32_t s = ld_relaxed(status + ((int64_t)l * tiles + j) * 256 + tid);
            const uint32_t flag = s & ~ST_CNT;
            if (flag == 0) {
                if (++spins > kSpinLimit) {
                    atomicOr(err, kErrSpin);
                    break;
                }
                if ((spins & 31u) == 0) __nanosleep(64);
                continue;
            }
            excl += s & ST_CNT;
            if (flag == ST_PRE) break;
            --j;
        }
        st_relaxed(my, ST_PRE | (excl + total));
    }
    gadd[tid] = base[((int64_t)l * passes + pass) * 256 + tid] + excl - tstart[tid];
    __syncthreads();

#pragma unroll
    for (int i = 0; i < SP_ITEMS; ++i) {
        const uint32_t d = dig[i];
        if (d < 256) {
            pos[i] += tstart[d] + whist[warp][d];
            sdig[pos[i]] = (uint8_t)d;
        }
    }
    __syncthreads();
    // Global destination of tile position s = tid + k * NT (digit runs are
    // contiguous), computed once for all components.
    uint32_t doff[SP_ITEMS];
#pragma unroll
    for (int k = 0; k < SP_ITEMS; ++k) {
        const int sp = tid + k * NT;
        doff[k] = sp < nvalid ? gadd[sdig[sp]] + (uint32_t)sp : 0u;
    }
    // Scatter each component (ids, then key words) through shared memory so
    // that the global writes of one digit run are contiguous; the next
    // component's loads are issued before the current one is written out.
    auto load_comp = [&](int comp, uint32_t (&v)[SP_ITEMS]) {
        const bool iota = comp == 0 && !vin;   // the first pass: an id is its position
        const uint32_t* src = iota ? kin : (comp == 0 ? vin : kin + (comp - 1) * LN) + seg + t0;
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i) {
            const int e = warp * (32 * SP_ITEMS) + i * 32 + lane;
            // the digit's own word is already in shared memory
            v[i] = dig[i] >= 256 ? 0u : iota ? (uint32_t)(t0 + e) : comp == word + 1 ? wtile[e] : src[e];
        }
    };
    uint32_t cur[SP_ITEMS];
    load_comp(0, cur);
    for (int comp = 0; comp <= KW; ++comp) {
        uint32_t* dst = (comp == 0 ? vout : kout + (comp - 1) * LN) + seg;
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i)
            if (dig[i] < 256) buf[pos[i]] = cur[i];
        if (comp < KW) load_comp(comp + 1, cur);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SP_ITEMS; ++k) {
            const int sp = tid + k * NT;
            if (sp < nvalid) dst[doff[k]] = buf[sp];
        }
        __syncthreads();
    }
}

// One digit pass over one-word keys. Each pair is read once into registers,
// ranked, exchanged through shared memory and written out; an exchanged pair's
// digit is taken from its key. k_sort_pass keeps a digit and a copy of the key
// per position and exchanges one component at a time: four passes over 16M
// pairs take 0.31 ms here, had taken 0.64 ms there, over 200M pairs 3.7 ms instead
// of 7.0 (3.3 TB/s). 4,096 pairs a tile and four blocks per SM: 512 threads x 8
// pairs 0.35 ms, x 16 0.33, 256 x 24 0.31, three blocks of 256 x 16 0.33, five
// 0.35 (they spill).
// vin null: a pair's id is its position (the first pass).
__global__ void __launch_bounds__(NT, 4) k_sort_pass_word(const uint32_t* __restrict__ kin,
                                                         const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
                                                         uint32_t* __restrict__ vout, int64_t N, int tiles, int shift,
                                                         const uint32_t* __restrict__ base, int passes, int pass,
                                                         uint32_t* status, uint32_t* counter, int* err) {
    static_assert(SP_WARPS * 768 * 4 <= SP_TILE * 8 && SP_ITEMS % 2 == 0, "counters and pairs share the buffer");
    __shared__ __align__(16) unsigned char raw[SP_TILE * 8];   // counters and masks, then the pairs
    uint32_t* whist = reinterpret_cast<uint32_t*>(raw);       // [SP_WARPS][256]
    __shared__ uint32_t gadd[256];
    __shared__ uint32_t ws[8];
    __shared__ uint32_t s_vb;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_vb = atomicAdd(counter, 1u);
    for (int i = tid; i < SP_WARPS * 192; i += NT) reinterpret_cast<uint4*>(raw)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t vb = s_vb;
    const int l = (int)(vb / (uint32_t)tiles), tile = (int)(vb % (uint32_t)tiles);
    const int64_t seg = (int64_t)l * N, t0 = (int64_t)tile * SP_TILE;
    const int nvalid = (N - t0 < SP_TILE) ? (int)(N - t0) : SP_TILE;
    const int e0 = warp * (32 * SP_ITEMS) + lane;
    kin += seg + t0;
    uint32_t key[SP_ITEMS], pos[SP_ITEMS];
    // Elements past the end carry the largest digit: last in the tile's order,
    // they end at the positions from nvalid on, which are not written out.
#pragma unroll
    for (int i = 0; i < SP_ITEMS; ++i) key[i] = e0 + i * 32 < nvalid ? kin[e0 + i * 32] : 0xFFFFFFFFu;
    // Stable ranks within the warp: element order is (item, lane).
    uint32_t* wh = whist + warp * 256;
    uint32_t* wm = whist + (SP_WARPS + 2 * warp) * 256;
#pragma unroll
    for (int i = 0; i < SP_ITEMS; i += 2)
        rank_two(wm, wh, (key[i] >> shift) & 255u, (key[i + 1] >> shift) & 255u, pos[i], pos[i + 1]);
    __syncthreads();
    // Thread tid owns digit tid: the tile's count and each warp's first position.
    uint32_t total = 0;
    uint32_t* my = status + ((int64_t)l * tiles + tile) * 256 + tid;
#pragma unroll
    for (int w = 0; w < SP_WARPS; ++w) total += whist[w * 256 + tid];
    const uint32_t live = tid == 255 ? total - (uint32_t)(SP_TILE - nvalid) : total;
    st_relaxed(my, (tile == 0 ? ST_PRE : ST_AGG) | live);
    const uint32_t start = block_excl_scan(total, ws, nullptr);
    uint32_t run = start;
#pragma unroll
    for (int w = 0; w < SP_WARPS; ++w) {
        const uint32_t c = whist[w * 256 + tid];
        whist[w * 256 + tid] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SP_ITEMS; ++i) pos[i] += wh[(key[i] >> shift) & 255u];
    __syncthreads();   // the counters are read: the buffer takes the pairs
    uint32_t* bk = reinterpret_cast<uint32_t*>(raw);
    uint32_t* bv = bk + SP_TILE;
    if (vin) {
        const uint32_t* vp = vin + seg + t0 + e0;
        uint32_t val[SP_ITEMS];
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i) val[i] = e0 + i * 32 < nvalid ? vp[i * 32] : 0u;
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i) bk[pos[i]] = key[i];
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i) bv[pos[i]] = val[i];
    } else {
#pragma unroll
        for (int i = 0; i < SP_ITEMS; ++i) {
            bk[pos[i]] = key[i];
            bv[pos[i]] = (uint32_t)(t0 + e0 + i * 32);
        }
    }
    // Decoupled look-back for digit tid, four predecessors at a time.
    uint32_t excl = 0;
    if (tile > 0) {
        int j = tile - 1;
        uint32_t spins = 0;
        bool done = false;
        while (!done) {
            uint32_t s[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                s[q] = j - q >= 0 ? ld_relaxed(my - (int64_t)(tile - j + q) * 256) : 0u;
            int used = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t flag = s[q] & ~ST_CNT;
                if (done || used < q || flag == 0) continue;
                excl += s[q] & ST_CNT;
                ++used;
                done = flag == ST_PRE;
            }
            j -= used;
            if (used == 0) {
                if (++spins > kSpinLimit) {
                    atomicOr(err, kErrSpin);
                    break;
                }
                if ((spins & 31u) == 0) __nanosleep(64);
            }
        }
        st_relaxed(my, ST_PRE | (excl + live));
    }
    gadd[tid] = base[((int64_t)l * passes + pass) * 256 + tid] + excl - start;
    __syncthreads();
    kout += seg;
    vout += seg;
#pragma unroll
    for (int k = 0; k < SP_ITEMS; ++k) {
        const int sp = tid + k * NT;
        if (sp < nvalid) {
            const uint32_t k0 = bk[sp], o = gadd[(k0 >> shift) & 255u] + (uint32_t)sp;
            kout[o] = k0;
            vout[o] = bv[sp];
        }
    }
}

// ---- Top-word-first ordering ----
// The digit passes can run over the key's top word alone (its leading 32
// bits), moving that word and the ids. The lower words stay in point order, as
// rows of lw words (1, 2 or 4), and are read through the ids where they are
// needed: each run of equal top words is ordered by (lower words, id) (the
// LSD passes leave a run's ids ascending, so this is the order the full sort
// produces), the run-length passes compare them inside such runs, and a
// bucket's key takes one row. Rows gathered into sorted order first, word by
// word, had cost 9.3 ms at 200M keys of four words.

// Lower words of point `id` of the table that starts at seg.
template <int KWL>
__device__ __forceinline__ void low_row(const uint32_t* __restrict__ low, int64_t seg, uint32_t id, uint32_t* e) {
    if constexpr (KWL == 1) {
        e[0] = __ldg(low + seg + id);
    } else if constexpr (KWL == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(low) + seg + id);
        e[0] = v.x;
        e[1] = v.y;
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(low) + seg + id);
        e[0] = v.x;
        e[1] = v.y;
        e[2] = v.z;
    }
}

// (lower words from the most significant down, then id) of a < of b
template <int KWL>
__device__ __forceinline__ bool run_less(const uint32_t (&a)[KWL + 1], const uint32_t (&b)[KWL + 1]) {
#pragma unroll
    for (int k = KWL - 1; k >= 0; --k)
        if (a[k] != b[k]) return a[k] < b[k];
    return a[KWL] < b[KWL];
}

// Marks sorted position i of table l as holding the same whole key as position
// i - 1 (words of 32 positions, tables padded to 4,096-position tiles: the
// layout of the boundary flags).
__device__ __forceinline__ void mark_same(uint32_t* same, int64_t N, int64_t l, int64_t i) {
    atomicOr(same + l * ((N + SP_TILE - 1) / SP_TILE * (SP_TILE / 32)) + (i >> 5), 1u << (i & 31));
}
template <int KWL>
__device__ __forceinline__ bool same_row(const uint32_t* a, const uint32_t* b) {
    bool eq = true;
#pragma unroll
    for (int k = 0; k < KWL; ++k) eq = eq && a[k] == b[k];
    return eq;
}

// Runs of two or more equal top words, found from their first element. Runs of
// two, by far the most where points fall nearly alone (of 200M positions of the
// 10M-point build more than the lists hold), are ordered here (by the thread
// that meets them: collected per block first, one to four pairs in flight a
// thread, the kernel takes 13 to 70 % longer); longer ones go to three lists:
// 3..8 (tiny), 9..32 (small), 33..kRunMax (large); a longer run or a full list
// sets cnt[3] (the caller then sorts all words instead).
// Block (x, table y) examines RUN_TILE positions from shared memory, one
// position in RUN_ITEMS rows per thread (consecutive threads, consecutive
// positions). List slots are claimed per block (shared counters, then one
// global atomic per block and class): with tens of thousands of runs per
// table, one global atomic per run or per warp serialises on the counters.
constexpr int RUN_ITEMS = 8;
constexpr int RUN_TILE = NT * RUN_ITEMS;
template <int KWL>
__global__ void __launch_bounds__(NT) k_run_find(const uint32_t* __restrict__ top, int64_t N,
                                                const uint32_t* __restrict__ low, uint32_t* __restrict__ ids,
                                                RunLists rl) {
    __shared__ unsigned int sc[3], sbase[3];
    __shared__ uint32_t w[RUN_TILE + 10];   // positions i0 - 1 .. i0 + RUN_TILE + 8
    const int64_t seg = (int64_t)blockIdx.y * N;
    const uint32_t* t = top + seg;
    const int64_t i0 = (int64_t)blockIdx.x * RUN_TILE;
    if (threadIdx.x < 3) sc[threadIdx.x] = 0;
    for (int j = threadIdx.x; j < RUN_TILE + 10; j += NT) {
        const int64_t i = i0 + j - 1;
        // past either end of the table: a value that differs from its neighbour
        if (i >= 0 && i < N) w[j] = t[i];
        else w[j] = ~t[i < 0 ? 0 : N - 1];
    }
    __syncthreads();
    uint32_t len[RUN_ITEMS];
    unsigned int mine[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < RUN_ITEMS; ++k) {
        const int j = k * NT + threadIdx.x + 1;
        const int64_t i = i0 + j - 1;
        const uint32_t v = w[j];
        uint32_t n = 1;
        if (i + 1 < N && w[j + 1] == v && w[j - 1] != v) {
            n = 2;
            while (n < 9 && i + n < N && w[j + n] == v) ++n;
            if (n == 9) {   // the words ascend: halve the rest
                if (i + kRunMax < N && t[i + kRunMax] == v) {
                    atomicOr(rl.cnt + 3, 1u);
                    n = 1;
                } else {
                    int64_t lo = i + 9, hi = min(N, i + kRunMax);   // hi: differs, or the end
                    while (lo < hi) {
                        const int64_t mid = (lo + hi) >> 1;
                        if (t[mid] == v) lo = mid + 1;
                        else hi = mid;
                    }
                    n = (uint32_t)(lo - i);
                }
            } else if (n == 2) {
                uint32_t a[KWL + 1], b[KWL + 1];
                a[KWL] = ids[seg + i];
                b[KWL] = ids[seg + i + 1];
                low_row<KWL>(low, seg, a[KWL], a);
                low_row<KWL>(low, seg, b[KWL], b);
                if (run_less<KWL>(b, a)) {
                    ids[seg + i] = b[KWL];
                    ids[seg + i + 1] = a[KWL];
                }
                if (same_row<KWL>(a, b)) mark_same(rl.same, N, blockIdx.y, i + 1);
            }
        }
        len[k] = n;
        mine[0] += (n > 2 && n <= 8) ? 1u : 0u;
        mine[1] += (n > 8 && n <= 32) ? 1u : 0u;
        mine[2] += n > 32 ? 1u : 0u;
    }
    unsigned int off[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) off[c] = mine[c] ? atomicAdd(&sc[c], mine[c]) : 0u;
    __syncthreads();
    if (threadIdx.x < 3) sbase[threadIdx.x] = sc[threadIdx.x] ? atomicAdd(rl.cnt + threadIdx.x, sc[threadIdx.x]) : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RUN_ITEMS; ++k) {
        const uint32_t n = len[k];
        if (n <= 2) continue;
        const int c = n <= 8 ? 0 : (n <= 32 ? 1 : 2);
        const unsigned int slot = sbase[c] + off[c]++;
        const unsigned int cap = c == 0 ? rl.tcap : (c == 1 ? rl.scap : rl.lcap);
        unsigned long long* pos = c == 0 ? rl.tpos : (c == 1 ? rl.spos : rl.lpos);
        uint32_t* lens = c == 0 ? rl.tlen : (c == 1 ? rl.slen : rl.llen);
        if (slot < cap) {
            pos[slot] = (unsigned long long)(seg + i0 + k * NT + threadIdx.x);
            lens[slot] = n;
        } else {
            atomicOr(rl.cnt + 3, 2u);
        }
    }
}

// One thread per run of 3 to 8: an odd-even transposition sort over eight
// register slots (missing slots hold all-ones, above every element).
template <int KWL>
__global__ void k_run_sort_tiny(const unsigned long long* __restrict__ tpos, const uint32_t* __restrict__ tlen,
                                const unsigned int* __restrict__ cnt, unsigned int tcap, int64_t N,
                                const uint32_t* __restrict__ low,
                                uint32_t* __restrict__ ids, uint32_t* __restrict__ same) {
    const unsigned int nrun = min(cnt[0], tcap);
    for (unsigned int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrun; r += gridDim.x * blockDim.x) {
        const int64_t pos = (int64_t)tpos[r];
        const int len = (int)tlen[r];
        const int64_t l = pos / N, seg = l * N;
        uint32_t e[8][KWL + 1];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
#pragma unroll
            for (int k = 0; k <= KWL; ++k) e[t][k] = 0xFFFFFFFFu;
            if (t < len) {
                e[t][KWL] = ids[pos + t];
                low_row<KWL>(low, seg, e[t][KWL], e[t]);
            }
        }
#pragma unroll
        for (int ph = 0; ph < 8; ++ph) {
#pragma unroll
            for (int t = ph & 1; t + 1 < 8; t += 2) {
                if (run_less<KWL>(e[t + 1], e[t])) {
#pragma unroll
                    for (int k = 0; k <= KWL; ++k) {
                        const uint32_t x = e[t][k];
                        e[t][k] = e[t + 1][k];
                        e[t + 1][k] = x;
                    }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            if (t < len) ids[pos + t] = e[t][KWL];
            if (t > 0 && t < len && same_row<KWL>(e[t], e[t - 1])) mark_same(same, N, l, pos - seg + t);
        }
    }
}

// One warp per run of at most 32: a bitonic sort across the lanes (missing
// lanes hold all-ones, above every element: ids are below 2^32 - 1).
template <int KWL>
__global__ void k_run_sort_small(const unsigned long long* __restrict__ spos, const uint32_t* __restrict__ slen,
                                 const unsigned int* __restrict__ cnt, unsigned int scap, int64_t N,
                                 const uint32_t* __restrict__ low,
                                uint32_t* __restrict__ ids, uint32_t* __restrict__ same) {
    const int lane = threadIdx.x & 31;
    const unsigned int nrun = min(cnt[1], scap);
    for (unsigned int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrun;
         r += (gridDim.x * blockDim.x) >> 5) {
        const int64_t pos = (int64_t)spos[r];
        const int len = (int)slen[r];
        const int64_t l = pos / N, seg = l * N;
        uint32_t e[KWL + 1];
#pragma unroll
        for (int k = 0; k <= KWL; ++k) e[k] = 0xFFFFFFFFu;
        if (lane < len) {
            e[KWL] = ids[pos + lane];
            low_row<KWL>(low, seg, e[KWL], e);
        }
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                uint32_t o[KWL + 1];
#pragma unroll
                for (int c = 0; c <= KWL; ++c) o[c] = __shfl_xor_sync(0xffffffffu, e[c], j);
                const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
                const bool o_less = run_less<KWL>(o, e);
                if (o_less == keep_min) {
#pragma unroll
                    for (int c = 0; c <= KWL; ++c) e[c] = o[c];
                }
            }
        }
        if (lane < len) ids[pos + lane] = e[KWL];
        uint32_t prev[KWL];
#pragma unroll
        for (int c = 0; c < KWL; ++c) prev[c] = __shfl_up_sync(0xffffffffu, e[c], 1);
        if (lane > 0 && lane < len && same_row<KWL>(e, prev)) mark_same(same, N, l, pos - seg + lane);
    }
}

// One block per run of 33 to kRunMax elements: a bitonic sort in shared memory.
template <int KWL>
__global__ void __launch_bounds__(NT) k_run_sort_large(const unsigned long long* __restrict__ lpos,
                                                      const uint32_t* __restrict__ llen,
                                                      const unsigned int* __restrict__ cnt, unsigned int lcap,
                                                      int64_t N, const uint32_t* __restrict__ low,
                                                      uint32_t* __restrict__ ids, uint32_t* __restrict__ same) {
    __shared__ uint32_t sv[KWL + 1][kRunMax];
    const unsigned int nrun = min(cnt[2], lcap);
    for (unsigned int r = blockIdx.x; r < nrun; r += gridDim.x) {
        const int64_t pos = (int64_t)lpos[r];
        const int len = (int)llen[r];
        const int64_t l = pos / N, seg = l * N;
        int n2 = 64;
        while (n2 < len) n2 <<= 1;
        for (int t = threadIdx.x; t < n2; t += NT) {
            uint32_t e[KWL + 1];
#pragma unroll
            for (int k = 0; k <= KWL; ++k) e[k] = 0xFFFFFFFFu;
            if (t < len) {
                e[KWL] = ids[pos + t];
                low_row<KWL>(low, seg, e[KWL], e);
            }
#pragma unroll
            for (int k = 0; k <= KWL; ++k) sv[k][t] = e[k];
        }
        __syncthreads();
        for (int k = 2; k <= n2; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int t = threadIdx.x; t < n2; t += NT) {
                    const int u = t ^ j;
                    if (u > t) {
                        uint32_t a[KWL + 1], b[KWL + 1];
#pragma unroll
                        for (int c = 0; c <= KWL; ++c) {
                            a[c] = sv[c][t];
                            b[c] = sv[c][u];
                        }
                        const bool asc = (t & k) == 0;
                        if (run_less<KWL>(b, a) == asc) {
#pragma unroll
                            for (int c = 0; c <= KWL; ++c) {
                                sv[c][t] = b[c];
                                sv[c][u] = a[c];
                            }
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int t = threadIdx.x; t < len; t += NT) {
            ids[pos + t] = sv[KWL][t];
            bool eq = t > 0;
#pragma unroll
            for (int c = 0; c < KWL; ++c) eq = eq && sv[c][t] == sv[c][t > 0 ? t - 1 : 0];
            if (eq) mark_same(same, N, l, pos - seg + t);
        }
        __syncthreads();
    }
}

// A point's lower key words (rows of lw words, as low_row; unused ones zero).
__device__ __forceinline__ uint4 low_words(const uint32_t* __restrict__ low, int lw, int64_t row) {
    if (lw == 1) return make_uint4(__ldg(low + row), 0u, 0u, 0u);
    if (lw == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(low) + row);
        return make_uint4(v.x, v.y, 0u, 0u);
    }
    return __ldg(reinterpret_cast<const uint4*>(low) + row);
}

// Bucket boundaries of one tile of 4,096 sorted positions: warp w takes positions
// [512 w, 512 w + 512) as 16 rows of 32 lanes. A position whose key differs
// from its predecessor's starts a bucket; flags gets one word per row, tile_cnt
// the tile's total. LOW: top-word-first form, keys = the sorted top words, flags
// hold the positions whose whole key equals the one before (looking up the lower
// words again had taken 1.65 ms at 200M positions, now 0.19). Otherwise keys =
// KW arrays of L*N words.
template <bool LOW>
__global__ void __launch_bounds__(NT) k_rl_count(SortedKeys s, int64_t N, int L, int KW, uint32_t* __restrict__ tile_cnt,
                                                 uint32_t* flags) {
    __shared__ uint32_t ws[SP_WARPS];
    const int l = blockIdx.y, tile = blockIdx.x, tiles = gridDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t LN = (int64_t)L * N, seg = (int64_t)l * N;
    const int64_t w0 = (int64_t)tile * SP_TILE + (int64_t)warp * (32 * SP_ITEMS);
    uint32_t* fl = flags + ((int64_t)l * tiles + tile) * (SP_TILE / 32) + warp * SP_ITEMS;
    const uint32_t marks = LOW && lane < SP_ITEMS ? fl[lane] : 0u;
    uint32_t mine = 0;
#pragma unroll
    for (int k0 = 0; k0 < SP_ITEMS; k0 += 4) {
        bool same[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int64_t i = w0 + (k0 + q) * 32 + lane;
            same[q] = i > 0 && i < N && s.keys[seg + i] == s.keys[seg + i - 1];
        }
        if constexpr (LOW) {
            // the runs' sorts marked the positions whose lower words are equal too
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t row = __shfl_sync(0xffffffffu, marks, k0 + q);   // by all lanes
                same[q] = same[q] && ((row >> lane) & 1u);
            }
        } else {
            for (int w = 1; w < KW; ++w)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (same[q]) {
                        const int64_t a = w * LN + seg + w0 + (k0 + q) * 32 + lane;
                        same[q] = s.keys[a] == s.keys[a - 1];
                    }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t ball = __ballot_sync(0xffffffffu, !same[q] && w0 + (k0 + q) * 32 + lane < N);
            if (lane == k0 + q) mine = ball;
        }
    }
    if (lane < SP_ITEMS) fl[lane] = mine;
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(mine));
    if (lane == 0) ws[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < SP_WARPS; ++w) tot += ws[w];
        tile_cnt[(int64_t)l * tiles + tile] = tot;
    }
}

__global__ void k_rl_scan(const uint32_t* __restrict__ tile_cnt, int tiles, uint32_t* __restrict__ tile_off,
                          uint32_t* __restrict__ nb) {
    __shared__ uint32_t ws[SP_WARPS];
    const int l = blockIdx.x;
    uint32_t carry = 0;
    for (int t0 = 0; t0 < tiles; t0 += NT) {
        const int t = t0 + threadIdx.x;
        const uint32_t v = t < tiles ? tile_cnt[(int64_t)l * tiles + t] : 0;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(v, ws, &tot);
        if (t < tiles) tile_off[(int64_t)l * tiles + t] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) nb[l] = carry;
}

// Bucket starts and unique keys at the positions that k_rl_count flagged, in
// order. LOW: four rows' lookups of lower words are in flight together (one
// after another they had taken 0.23 ms for 16M buckets, now 0.11).
template <bool LOW>
__global__ void __launch_bounds__(NT) k_rl_write(SortedKeys s, int64_t N, int L, int KW,
                                                 const uint32_t* __restrict__ flags, const uint32_t* __restrict__ tile_off,
                                                 const uint64_t* __restrict__ boff, uint32_t* __restrict__ starts,
                                                 uint32_t* __restrict__ ukeys) {
    __shared__ uint32_t ws[SP_WARPS];
    const int l = blockIdx.y, tile = blockIdx.x, tiles = gridDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t LN = (int64_t)L * N, seg = (int64_t)l * N;
    const int64_t w0 = (int64_t)tile * SP_TILE + (int64_t)warp * (32 * SP_ITEMS);
    const uint32_t mine =
        lane < SP_ITEMS ? flags[((int64_t)l * tiles + tile) * (SP_TILE / 32) + warp * SP_ITEMS + lane] : 0u;
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(mine));
    if (lane == 0) ws[warp] = c;
    __syncthreads();
    uint64_t g = boff[l] + tile_off[(int64_t)l * tiles + tile];
    for (int w = 0; w < warp; ++w) g += ws[w];
    const uint32_t below = (1u << lane) - 1u;
#pragma unroll
    for (int k0 = 0; k0 < SP_ITEMS; k0 += 4) {
        uint32_t ball[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) ball[q] = __shfl_sync(0xffffffffu, mine, k0 + q);
        if constexpr (LOW) {
            uint32_t id[4], top[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t a = seg + w0 + (k0 + q) * 32 + lane;
                const bool f = (ball[q] >> lane) & 1u;
                id[q] = f ? s.ids[a] : 0u;
                top[q] = f ? s.keys[a] : 0u;
            }
            uint4 x[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[q] = make_uint4(0, 0, 0, 0);
                if ((ball[q] >> lane) & 1u) x[q] = low_words(s.low, s.lw, seg + id[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if ((ball[q] >> lane) & 1u) {
                    const uint64_t o = g + __popc(ball[q] & below);
                    starts[o] = (uint32_t)(w0 + (k0 + q) * 32 + lane);
                    if (s.lw == 1) {
                        reinterpret_cast<uint2*>(ukeys)[o] = make_uint2(x[q].x, top[q]);
                    } else if (s.lw == 2) {
                        ukeys[o * 3] = x[q].x;
                        ukeys[o * 3 + 1] = x[q].y;
                        ukeys[o * 3 + 2] = top[q];
                    } else {
                        reinterpret_cast<uint4*>(ukeys)[o] = make_uint4(x[q].x, x[q].y, x[q].z, top[q]);
                    }
                }
                g += __popc(ball[q]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if ((ball[q] >> lane) & 1u) {
                    const int64_t i = w0 + (k0 + q) * 32 + lane;
                    const uint64_t o = g + __popc(ball[q] & below);
                    starts[o] = (uint32_t)i;
                    for (int w = 0; w < KW; ++w) ukeys[o * KW + w] = s.keys[w * LN + seg + i];
                }
                g += __popc(ball[q]);
            }
        }
    }
}

// Finished lookup hashes of ITEMS keys of table l (indices j0 + i * NTH, clamped
// to the last). Fields are contiguous from column M - 1's offset upwards and
// their widths the same for every thread: they are taken from a 64-bit window
// (a 128-bit shift per field had been most of the kernel's instructions).
template <bool WIDE, int NTH, int ITEMS>
__device__ __forceinline__ void key_hashes(const HashBuild& h, int l, uint64_t bo, int64_t B, int64_t j0,
                                           uint64_t (&hh)[ITEMS]) {
    const int M = h.M, KW = h.KW;
    if constexpr (WIDE) {   // KW > 4
#pragma unroll 1
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t* key = h.ukeys + (bo + min(j0 + i * NTH, B - 1)) * KW;
            uint64_t hs = 0;
            for (int m = 0; m < M; ++m) {
                const int c = l * M + m;
                hs += (uint64_t)key_get(key, __ldg(h.foff + c), __ldg(h.fbits + c)) * __ldg(h.rmul + c);
            }
#pragma unroll
            for (int q = 0; q < ITEMS; ++q) hh[q] = q == i ? hash_finish(hs) : hh[q];
        }
    } else {
        uint32_t k[4][ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t* key = h.ukeys + (bo + min(j0 + i * NTH, B - 1)) * KW;
#pragma unroll
            for (int w = 0; w < 4; ++w) k[w][i] = w < KW ? __ldg(key + w) : 0u;
        }
        const int pos = __ldg(h.foff + (int64_t)l * M + M - 1);
        int w = pos >> 5;
        uint64_t win[ITEMS];
        auto word = [&](int i) { return w == 0 ? k[0][i] : w == 1 ? k[1][i] : w == 2 ? k[2][i] : w == 3 ? k[3][i] : 0u; };
        int have = 32 - (pos & 31);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            win[i] = word(i) >> (pos & 31);
            hh[i] = 0;
        }
        for (int m = M - 1; m >= 0; --m) {
            const int c = l * M + m;
            const int bits = __ldg(h.fbits + c);
            if (bits == 0) continue;
            const uint64_t mul = __ldg(h.rmul + c);
            if (have < bits) {
                ++w;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) win[i] |= (uint64_t)word(i) << have;
                have += 32;
            }
            const uint32_t mask = bits == 32 ? 0xFFFFFFFFu : (1u << bits) - 1u;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                hh[i] += (uint64_t)((uint32_t)win[i] & mask) * mul;
                win[i] >>= bits;
            }
            have -= bits;
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) hh[i] = hash_finish(hh[i]);
    }
}

// Sizes of buckets j0 + i * NTH of a table, and the largest of the block's with
// one atomic (one per warp serialises on the single address).
template <int NTH, int ITEMS>
__device__ __forceinline__ void bucket_sizes(const HashBuild& h, uint64_t bo, int64_t B, int64_t j0) {
    __shared__ uint32_t smax[NTH / 32];
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int64_t j = j0 + i * NTH;
        if (j >= B) break;
        const uint32_t end = j + 1 < B ? h.starts[bo + j + 1] : (uint32_t)h.N;
        const uint32_t sz = end - h.starts[bo + j];
        h.sizes[bo + j] = sz;
        mx = max(mx, sz);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NTH / 32; ++w) mx = max(mx, smax[w]);
        atomicMax(h.max_size, mx);
    }
}

// Claims the first empty slot in probe order from group g on (a group's slots
// in order, then the next group), then stores the bucket index beside it; cur
// is the first group's fingerprint word as last seen. Lookups stop at the first
// empty slot they meet, which can only lie past every key inserted along the
// same path.
__device__ __forceinline__ void hash_insert(unsigned long long* slots, uint32_t gmask, uint32_t g, uint32_t fp, uint32_t j,
                                            unsigned long long cur, int* err) {
    for (uint32_t p = 0; p <= gmask; ++p) {
        unsigned long long* grp = slots + (uint64_t)((g + p) & gmask) * kGroupWords;
        if (p > 0) cur = *reinterpret_cast<volatile unsigned long long*>(grp);
        // One 64-bit CAS per attempt on the group's fingerprint word; each
        // failure means another insert took a slot, so at most four tries.
        for (int tries = 0; tries <= kGroupSlots; ++tries) {
            int e = 0;
            while (e < kGroupSlots && ((cur >> (16 * e)) & 0xFFFFu) != kEmptyFp) ++e;
            if (e == kGroupSlots) break;   // group full: next group
            const unsigned long long nw = (cur & ~(0xFFFFull << (16 * e))) | ((unsigned long long)fp << (16 * e));
            const unsigned long long old = atomicCAS(grp, cur, nw);
            if (old == cur) {
                reinterpret_cast<uint32_t*>(grp + 1)[e] = j;
                return;
            }
            cur = old;
        }
    }
    atomicOr(err, kErrHashFull);
}

// Key by key in place. The first attempt takes the home group for empty, as
// most are, without reading it, two keys' attempts in flight per thread (16M
// keys in tables of 17 MB: 0.43 ms with the sizes; reading the group first 0.54,
// one key per thread 0.48, four 0.48).
constexpr int HB_ITEMS = 2;
template <bool WIDE>
__global__ void __launch_bounds__(NT) k_hash_build(HashBuild h) {
    const int l = blockIdx.y;
    const int64_t j0 = (int64_t)blockIdx.x * (NT * HB_ITEMS) + threadIdx.x;
    const uint64_t bo = h.boff[l];
    const int64_t B = (int64_t)(h.boff[l + 1] - bo);
    if ((int64_t)blockIdx.x * (NT * HB_ITEMS) >= B) return;
    const uint32_t gmask = h.hmask[l];
    uint64_t hh[HB_ITEMS];
    key_hashes<WIDE, NT, HB_ITEMS>(h, l, bo, B, j0, hh);
    uint32_t* fl = h.filt + h.fl_off[l];
    const uint32_t fmask = h.fl_mask[l];
    unsigned long long* slots = h.hslots + h.hoff[l];
    constexpr unsigned long long kEmptyGroup = ~0ull;
    unsigned long long got[HB_ITEMS];
#pragma unroll
    for (int i = 0; i < HB_ITEMS; ++i)
        if (j0 + i * NT < B) atomicOr(fl + (filter_word(hh[i]) & fmask), filter_bits(hh[i]));
#pragma unroll
    for (int i = 0; i < HB_ITEMS; ++i) {
        got[i] = kEmptyGroup;
        if (j0 + i * NT < B)
            got[i] = atomicCAS(slots + (uint64_t)((uint32_t)hh[i] & gmask) * kGroupWords, kEmptyGroup,
                               (kEmptyGroup & ~0xFFFFull) | slot_fp(hh[i]));
    }
#pragma unroll
    for (int i = 0; i < HB_ITEMS; ++i) {
        const int64_t j = j0 + i * NT;
        if (j >= B) break;
        const uint32_t g = (uint32_t)hh[i] & gmask;
        if (got[i] == kEmptyGroup) reinterpret_cast<uint32_t*>(slots + (uint64_t)g * kGroupWords + 1)[0] = (uint32_t)j;
        else hash_insert(slots, gmask, g, slot_fp(hh[i]), (uint32_t)j, got[i], h.err);
    }
    if (h.sizes) bucket_sizes<NT, HB_ITEMS>(h, bo, B, j0);
}

// By parts: k_hash_split orders the keys of a tile by the part of the table
// (kHashPartGroups groups) that their home group lies in and appends them to
// the parts' records; k_hash_fill builds a part and its filter words in shared
// memory and writes them out whole. In place, a key cost three random accesses
// of L2 or, in tables beyond its size, of memory, and the tables had to be
// cleared first: 0.66 ms for 16M keys in 16 tables, clearing and sizes included,
// against 0.38 now; 9.1 ms for 200M in 20 tables, now 5.4. 512 threads x 16 keys
// a tile: x 8 takes 0.20 instead of 0.23 ms at 16M but 4.1 instead of 3.7 at
// 200M, whose 4,096 parts leave a tile two keys a part.
// A record: bucket in the low half; group within the part (11 bits),
// fingerprint (16) and the filter bit outside it (5) in the high one.
constexpr int HS_T = 512, HS_ITEMS = 16, HS_TILE = HS_T * HS_ITEMS;
static_assert(kHashPartGroups == 2048 && HS_TILE <= 8192 && kHashMaxParts <= 4096, "bit fields of a record and of a rank");
constexpr size_t hash_split_smem(uint32_t parts) { return (size_t)HS_TILE * 10 + (size_t)parts * 8; }

// A key that its part cannot take is listed; past the list's end it is only
// counted, and the caller of the form, who reads the count, builds in place.
__device__ __forceinline__ void hash_spill(const HashBuild& h, uint32_t* cnt, int l, uint32_t j) {
    const uint32_t s = atomicAdd(cnt, 1u);
    if (s < h.spill_cap) h.spill[s] = make_uint2((uint32_t)l, j);
}

__global__ void __launch_bounds__(HS_T, 2) k_hash_split(HashBuild h, uint32_t parts) {
    extern __shared__ __align__(16) unsigned char raw[];
    unsigned long long* buf = reinterpret_cast<unsigned long long*>(raw);              // [HS_TILE]
    uint16_t* bin = reinterpret_cast<uint16_t*>(raw + (size_t)HS_TILE * 8);            // [HS_TILE]
    uint32_t* hist = reinterpret_cast<uint32_t*>(raw + (size_t)HS_TILE * 10);          // [parts] counts, then starts
    uint32_t* gpos = hist + parts;                                                     // [parts] record of position 0
    __shared__ uint32_t ws[HS_T / 32];
    const int l = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t bo = h.boff[l];
    const int64_t B = (int64_t)(h.boff[l + 1] - bo), t0 = (int64_t)blockIdx.x * HS_TILE;
    if (t0 >= B) return;
    const uint32_t gmask = h.hmask[l];
    const uint32_t my_parts = gmask / kHashPartGroups + 1;
    for (uint32_t i = tid; i < my_parts; i += HS_T) hist[i] = 0;
    __syncthreads();
    uint32_t hi[HS_ITEMS], br[HS_ITEMS];   // record's high half; part and rank within it
#pragma unroll
    for (int i0 = 0; i0 < HS_ITEMS; i0 += 4) {
        uint64_t hh[4];
        key_hashes<false, HS_T, 4>(h, l, bo, B, t0 + i0 * HS_T + tid, hh);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t g = (uint32_t)hh[i] & gmask, part = g / kHashPartGroups;
            hi[i0 + i] = (g % kHashPartGroups) | (slot_fp(hh[i]) << 11) | ((uint32_t)(hh[i] >> 43) << 27);
            br[i0 + i] = 0;
            if (t0 + (i0 + i) * HS_T + tid < B) br[i0 + i] = (part << 16) | atomicAdd(hist + part, 1u);
        }
    }
    __syncthreads();
    // starts of the parts within the tile, and their places among the records
    const uint32_t per = (my_parts + HS_T - 1) / HS_T;
    uint32_t sum = 0;
    for (uint32_t q = 0; q < per; ++q) {
        const uint32_t b = tid * per + q;
        if (b < my_parts) sum += hist[b];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    uint32_t start = x - sum;
    for (int w = 0; w < warp; ++w) start += ws[w];
    for (uint32_t q = 0; q < per; ++q) {
        const uint32_t b = tid * per + q;
        if (b >= my_parts) break;
        const uint32_t c = hist[b];
        hist[b] = start;
        if (c) gpos[b] = atomicAdd(h.part_cnt + (size_t)l * parts + b, c) - start;
        start += c;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < HS_ITEMS; ++i) {
        const int64_t j = t0 + i * HS_T + tid;
        if (j < B) {
            const uint32_t part = br[i] >> 16, at = hist[part] + (br[i] & 0xFFFFu);
            buf[at] = ((unsigned long long)hi[i] << 32) | (uint32_t)j;
            bin[at] = (uint16_t)part;
        }
    }
    __syncthreads();
    const int n = (int)min((int64_t)HS_TILE, B - t0);
    for (int sp = tid; sp < n; sp += HS_T) {
        const uint32_t part = bin[sp], at = gpos[part] + (uint32_t)sp;
        if (at < h.part_cap) h.rec[((size_t)l * parts + part) * kHashPartCap + at] = buf[sp];
        else hash_spill(h, h.part_cnt + (size_t)h.L * parts, l, (uint32_t)buf[sp]);
    }
    bucket_sizes<HS_T, HS_ITEMS>(h, bo, B, t0 + tid);
}

__global__ void __launch_bounds__(NT) k_hash_fill(HashBuild h, uint32_t parts) {
    extern __shared__ __align__(16) unsigned char raw[];
    unsigned long long* fps = reinterpret_cast<unsigned long long*>(raw);              // [groups]
    uint4* idx = reinterpret_cast<uint4*>(raw + (size_t)kHashPartGroups * 8);          // [groups]
    uint32_t* fw = reinterpret_cast<uint32_t*>(raw + (size_t)kHashPartGroups * 24);    // [groups / 2]
    const int l = blockIdx.y, tid = threadIdx.x;
    const uint32_t gmask = h.hmask[l], part = blockIdx.x;
    const uint32_t my_parts = gmask / kHashPartGroups + 1;
    if (part >= my_parts) return;
    const uint32_t groups = min(gmask + 1, kHashPartGroups), words = max(groups / 2, 1u);
    for (uint32_t i = tid; i < groups; i += NT) {
        fps[i] = ~0ull;
        idx[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
    for (uint32_t i = tid; i < words; i += NT) fw[i] = 0u;
    __syncthreads();
    const size_t base = (size_t)l * parts + part;
    const unsigned long long* rec = h.rec + base * kHashPartCap;
    const uint32_t n = min(h.part_cnt[base], h.part_cap);
    for (uint32_t i0 = tid; i0 < n; i0 += 4 * NT) {
        unsigned long long r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = i0 + q * NT < n ? __ldcs(rec + i0 + q * NT) : 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (i0 + q * NT >= n) break;
            const uint32_t hi = (uint32_t)(r[q] >> 32), fp = (hi >> 11) & 0xFFFFu;
            uint32_t g = hi & (kHashPartGroups - 1);
            // filter_bits: bit 43.. of the hash, and bit 5 of the fingerprint on
            atomicOr(fw + (g >> 1), (1u << (hi >> 27)) | (1u << ((fp >> 5) & 31u)));
            bool in = false;
            for (uint32_t p = 0; p < groups && !in; ++p) {
                unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(fps + g);
                for (int tries = 0; tries <= kGroupSlots; ++tries) {
                    int e = 0;
                    while (e < kGroupSlots && ((cur >> (16 * e)) & 0xFFFFu) != kEmptyFp) ++e;
                    if (e == kGroupSlots) break;
                    const unsigned long long nw = (cur & ~(0xFFFFull << (16 * e))) | ((unsigned long long)fp << (16 * e));
                    const unsigned long long old = atomicCAS(fps + g, cur, nw);
                    if (old == cur) {
                        reinterpret_cast<uint32_t*>(idx + g)[e] = (uint32_t)r[q];
                        in = true;
                        break;
                    }
                    cur = old;
                }
                // the next group; past a part's last one, the insertion in place
                if (++g == groups) {
                    if (my_parts > 1) break;
                    g = 0;
                }
            }
            if (!in) hash_spill(h, h.part_cnt + (size_t)h.L * parts, l, (uint32_t)r[q]);
        }
    }
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(h.hslots + h.hoff[l] + (size_t)part * kHashPartGroups * kGroupWords);
    for (uint32_t i = tid; i < 2 * groups; i += NT) {
        const uint4 ix = idx[i >> 1];
        const unsigned long long f = fps[i >> 1];
        out[i] = i & 1 ? make_uint4(ix.z, ix.w, ~0u, ~0u) : make_uint4((uint32_t)f, (uint32_t)(f >> 32), ix.x, ix.y);
    }
    uint32_t* fo = h.filt + h.fl_off[l] + (size_t)part * (kHashPartGroups / 2);
    for (uint32_t i = tid; i < words; i += NT) fo[i] = fw[i];
}

// The spilled keys, in place once every part is written.
__global__ void k_hash_spilled(HashBuild h, uint32_t parts) {
    const uint32_t n = min(h.part_cnt[(size_t)h.L * parts], h.spill_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 s = h.spill[i];
        const int l = (int)s.x;
        const uint64_t bo = h.boff[l];
        uint64_t hh[1];
        key_hashes<false, 1, 1>(h, l, bo, (int64_t)(h.boff[l + 1] - bo), (int64_t)s.y, hh);
        const uint32_t gmask = h.hmask[l], g = (uint32_t)hh[0] & gmask;
        atomicOr(h.filt + h.fl_off[l] + (filter_word(hh[0]) & h.fl_mask[l]), filter_bits(hh[0]));
        unsigned long long* slots = h.hslots + h.hoff[l];
        hash_insert(slots, gmask, g, slot_fp(hh[0]), s.y,
                    *reinterpret_cast<volatile unsigned long long*>(slots + (uint64_t)g * kGroupWords), h.err);
    }
}

__global__ void k_decode_codes(const uint64_t* __restrict__ boff, const uint32_t* __restrict__ ukeys, int M, int KW,
                               const int32_t* __restrict__ cmin, const uint8_t* __restrict__ fbits,
                               const uint16_t* __restrict__ foff, float* __restrict__ codes) {
    const int l = blockIdx.y;
    const int64_t j = (int64_t)blockIdx.x * NT + threadIdx.x;
    const int64_t B = (int64_t)(boff[l + 1] - boff[l]);
    if (j >= B) return;
    uint32_t k[kMaxKW];
    for (int w = 0; w < KW; ++w) k[w] = ukeys[(boff[l] + j) * KW + w];
    float* out = codes + boff[l] * M;
    for (int m = 0; m < M; ++m) {
        const int c = l * M + m;
        out[(int64_t)m * B + j] = (float)(int32_t)(key_get(k, foff[c], fbits[c]) + (uint32_t)cmin[c]);
    }
}

__global__ void k_codes_minmax(const uint64_t* __restrict__ boff, const float* __restrict__ codes, int M,
                               int32_t* __restrict__ cmin, int32_t* __restrict__ cmax, int* err) {
    __shared__ int32_t slo[SP_WARPS], shi[SP_WARPS];
    const int l = blockIdx.y;
    const int64_t j = (int64_t)blockIdx.x * NT + threadIdx.x;
    const int64_t B = (int64_t)(boff[l + 1] - boff[l]);
    if ((int64_t)blockIdx.x * NT >= B) return;  // whole block idle: uniform exit
    const float* in = codes + boff[l] * M;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int m = 0; m < M; ++m) {
        int32_t lo = INT_MAX, hi = INT_MIN;
        if (j < B) {
            const float f = in[(int64_t)m * B + j];
            if (!(f == floorf(f) && f >= -2147483648.0f && f < 2147483648.0f)) {
                atomicOr(err, kErrNotIntegral);
            } else {
                lo = hi = (int32_t)f;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            slo[w] = lo;
            shi[w] = hi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < SP_WARPS; ++k) {
                lo = min(lo, slo[k]);
                hi = max(hi, shi[k]);
            }
            atomicMin(&cmin[l * M + m], lo);
            atomicMax(&cmax[l * M + m], hi);
        }
        __syncthreads();
    }
}

__global__ void k_pack_from_codes(const uint64_t* __restrict__ boff, const float* __restrict__ codes, int M, int KW,
                                  const int32_t* __restrict__ cmin, const uint8_t* __restrict__ fbits,
                                  const uint16_t* __restrict__ foff, uint32_t* __restrict__ ukeys) {
    const int l = blockIdx.y;
    const int64_t j = (int64_t)blockIdx.x * NT + threadIdx.x;
    const int64_t B = (int64_t)(boff[l + 1] - boff[l]);
    if (j >= B) return;
    const float* in = codes + boff[l] * M;
    uint32_t k[kMaxKW];
#pragma unroll
    for (int w = 0; w < kMaxKW; ++w) k[w] = 0;
    for (int m = 0; m < M; ++m) {
        const int c = l * M + m;
        if (fbits[c]) key_put(k, foff[c], fbits[c], (uint32_t)((int32_t)in[(int64_t)m * B + j] - cmin[c]));
    }
    for (int w = 0; w < KW; ++w) ukeys[(boff[l] + j) * KW + w] = k[w];
}

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as
// easy as 1, 2, 3", SC 2011), keyed by the seed, counter = element index.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

__global__ void k_random(float* __restrict__ A, float* __restrict__ u, int64_t nA, int64_t nu,
                         unsigned long long seed) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    if (i < nA) {
        const uint4 r = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 0u, 0u), key);
        const float u1 = ((r.x >> 8) + 1u) * (1.0f / 16777216.0f);   // (0, 1]
        const float u2 = (r.y >> 8) * (1.0f / 16777216.0f);          // [0, 1)
        A[i] = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);          // Box-Muller
    }
    if (i < nu) {
        const uint4 r = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 1u, 0u), key);
        u[i] = ((r.x >> 8) + 1u) * (1.0f / 16777216.0f);
    }
}

inline int blocks_for(int64_t n) { return (int)((n + NT - 1) / NT); }

}  // namespace

cudaError_t launch_pack_keys(const int32_t* codes, int64_t N, int L, int M, int KW, const int32_t* cmin,
                             const uint8_t* fbits, const uint16_t* foff, uint32_t* keys, uint32_t* vals,
                             uint32_t* low, int lw, cudaStream_t st) {
    const dim3 grid((unsigned)((N + NT * PK_ITEMS - 1) / (NT * PK_ITEMS)), (unsigned)L);
    if (KW > 4) k_pack_keys<true><<<grid, NT, 0, st>>>(codes, N, L, M, KW, cmin, fbits, foff, keys, vals, nullptr, 0);
    else k_pack_keys<false><<<grid, NT, 0, st>>>(codes, N, L, M, KW, cmin, fbits, foff, keys, vals, low, lw);
    return cudaGetLastError();
}

size_t sort_status_words(int64_t N, int L) {
    const int64_t tiles = (N + SP_TILE - 1) / SP_TILE;
    return (size_t)(L * tiles * 256 + 32);
}

cudaError_t run_segmented_sort(SortBuffers& sb, int64_t N, int L, int KW, int passes, int first_pass,
                               bool* result_in_alt, cudaStream_t st) {
    *result_in_alt = false;
    if (passes <= first_pass || N <= 1) return cudaSuccess;
    const int tiles = (int)((N + SP_TILE - 1) / SP_TILE);
    cudaError_t e;
    if ((e = cudaMemsetAsync(sb.hist, 0, sizeof(uint32_t) * L * passes * 256, st)) != cudaSuccess) return e;
    const dim3 hg((unsigned)((N + HIST_CHUNK - 1) / HIST_CHUNK), L);
    k_sort_hist<<<hg, NT, passes * 256 * sizeof(uint32_t), st>>>(sb.keys[0], N, L, passes, sb.hist);
    k_sort_digit_base<<<L * passes, NT, 0, st>>>(sb.hist, sb.base);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int cur = 0;
    const size_t status_words = sort_status_words(N, L);
    uint32_t* counter = sb.status + (status_words - 32);
    for (int p = first_pass; p < passes; ++p) {
        if ((e = cudaMemsetAsync(sb.status, 0, sizeof(uint32_t) * status_words, st)) != cudaSuccess) break;
        const uint32_t* vin = p == first_pass ? nullptr : sb.vals[cur];
        if (KW == 1)
            k_sort_pass_word<<<(unsigned)(L * tiles), NT, 0, st>>>(sb.keys[cur], vin, sb.keys[cur ^ 1], sb.vals[cur ^ 1],
                                                                   N, tiles, p * 8, sb.base, passes, p, sb.status,
                                                                   counter, sb.err);
        else
            k_sort_pass<<<(unsigned)(L * tiles), NT, 0, st>>>(sb.keys[cur], vin, sb.keys[cur ^ 1], sb.vals[cur ^ 1], N, L,
                                                              KW, tiles, p >> 2, (p & 3) * 8, sb.base, passes, p,
                                                              sb.status, counter, sb.err);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        cur ^= 1;
    }
    *result_in_alt = cur == 1;
    return e;
}

cudaError_t launch_run_find(const uint32_t* top, int64_t N, int L, int KW, const uint32_t* low, uint32_t* ids,
                            const RunLists& rl, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(rl.cnt, 0, 4 * sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(rl.same, 0, sizeof(uint32_t) * (size_t)L * ((N + SP_TILE - 1) / SP_TILE) * (SP_TILE / 32), st);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((N + RUN_TILE - 1) / RUN_TILE), (unsigned)L);
    switch (KW - 1) {
    case 1: k_run_find<1><<<grid, NT, 0, st>>>(top, N, low, ids, rl); break;
    case 2: k_run_find<2><<<grid, NT, 0, st>>>(top, N, low, ids, rl); break;
    case 3: k_run_find<3><<<grid, NT, 0, st>>>(top, N, low, ids, rl); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <int KWL>
void launch_run_sorts_w(const RunLists& rl, int64_t LN, int64_t N, const uint32_t* low, uint32_t* ids, cudaStream_t st) {
    // the lists' lengths stay on the device: grids for a full device, or fewer
    // where the keys cannot hold as many runs
    const unsigned gt = (unsigned)std::min<int64_t>((LN / 3 + NT - 1) / NT + 1, 152 * 16);
    const unsigned gs = (unsigned)std::min<int64_t>((LN / 9 * 32 + NT - 1) / NT + 1, 152 * 16);
    const unsigned gl = (unsigned)std::min<int64_t>(LN / 33 + 1, 152 * 4);
    k_run_sort_tiny<KWL><<<gt, NT, 0, st>>>(rl.tpos, rl.tlen, rl.cnt, rl.tcap, N, low, ids, rl.same);
    k_run_sort_small<KWL><<<gs, NT, 0, st>>>(rl.spos, rl.slen, rl.cnt, rl.scap, N, low, ids, rl.same);
    k_run_sort_large<KWL><<<gl, NT, 0, st>>>(rl.lpos, rl.llen, rl.cnt, rl.lcap, N, low, ids, rl.same);
}

cudaError_t launch_run_sorts(const RunLists& rl, int64_t N, int L, int KW, const uint32_t* low, uint32_t* ids,
                             cudaStream_t st) {
    const int64_t LN = (int64_t)L * N;
    switch (KW - 1) {
    case 1: launch_run_sorts_w<1>(rl, LN, N, low, ids, st); break;
    case 2: launch_run_sorts_w<2>(rl, LN, N, low, ids, st); break;
    case 3: launch_run_sorts_w<3>(rl, LN, N, low, ids, st); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_rl_count(const SortedKeys& keys, int64_t N, int L, int KW, uint32_t* tile_cnt, uint32_t* tile_off,
                            uint32_t* flags, uint32_t* nb, cudaStream_t st) {
    const int tiles = (int)((N + SP_TILE - 1) / SP_TILE);
    if (keys.low) k_rl_count<true><<<dim3(tiles, L), NT, 0, st>>>(keys, N, L, KW, tile_cnt, flags);
    else k_rl_count<false><<<dim3(tiles, L), NT, 0, st>>>(keys, N, L, KW, tile_cnt, flags);
    k_rl_scan<<<L, NT, 0, st>>>(tile_cnt, tiles, tile_off, nb);
    return cudaGetLastError();
}

cudaError_t launch_rl_write(const SortedKeys& keys, int64_t N, int L, int KW, const uint32_t* flags,
                            const uint32_t* tile_off, const uint64_t* boff, uint32_t* starts, uint32_t* ukeys,
                            cudaStream_t st) {
    const int tiles = (int)((N + SP_TILE - 1) / SP_TILE);
    if (keys.low) k_rl_write<true><<<dim3(tiles, L), NT, 0, st>>>(keys, N, L, KW, flags, tile_off, boff, starts, ukeys);
    else k_rl_write<false><<<dim3(tiles, L), NT, 0, st>>>(keys, N, L, KW, flags, tile_off, boff, starts, ukeys);
    return cudaGetLastError();
}

cudaError_t launch_hash_build(const HashBuild& h, cudaStream_t st) {
    if (h.maxB <= 0) return cudaSuccess;
    const dim3 grid((unsigned)((h.maxB + NT * HB_ITEMS - 1) / (NT * HB_ITEMS)), h.L);
    if (h.KW > 4) k_hash_build<true><<<grid, NT, 0, st>>>(h);
    else k_hash_build<false><<<grid, NT, 0, st>>>(h);
    return cudaGetLastError();
}

cudaError_t launch_hash_build_parts(const HashBuild& h, cudaStream_t st) {
    const uint32_t parts = std::max(h.max_groups / kHashPartGroups, 1u);
    const int split = (int)hash_split_smem(parts), fill = (int)kHashPartGroups * 26;
    static std::atomic<size_t> opted_split{0}, opted_fill{0};
    cudaError_t e = opt_in_smem(k_hash_split, (size_t)split, opted_split);
    if (e != cudaSuccess) return e;
    if ((e = opt_in_smem(k_hash_fill, (size_t)fill, opted_fill)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(h.part_cnt, 0, sizeof(uint32_t) * ((size_t)h.L * parts + 1), st)) != cudaSuccess) return e;
    k_hash_split<<<dim3((unsigned)((h.maxB + HS_TILE - 1) / HS_TILE), h.L), HS_T, split, st>>>(h, parts);
    k_hash_fill<<<dim3(parts, h.L), NT, fill, st>>>(h, parts);
    k_hash_spilled<<<152, NT, 0, st>>>(h, parts);
    return cudaGetLastError();
}

cudaError_t launch_decode_codes(const uint64_t* boff, const uint32_t* ukeys, int L, int M, int KW, int64_t maxB,
                                const int32_t* cmin, const uint8_t* fbits, const uint16_t* foff, float* codes,
                                cudaStream_t st) {
    if (maxB <= 0) return cudaSuccess;
    k_decode_codes<<<dim3(blocks_for(maxB), L), NT, 0, st>>>(boff, ukeys, M, KW, cmin, fbits, foff, codes);
    return cudaGetLastError();
}

cudaError_t launch_codes_minmax(const uint64_t* boff, const float* codes, int L, int M, int64_t maxB,
                                int32_t* cmin, int32_t* cmax, int* err, cudaStream_t st) {
    if (maxB <= 0) return cudaSuccess;
    k_codes_minmax<<<dim3(blocks_for(maxB), L), NT, 0, st>>>(boff, codes, M, cmin, cmax, err);
    return cudaGetLastError();
}

cudaError_t launch_pack_from_codes(const uint64_t* boff, const float* codes, int L, int M, int KW, int64_t maxB,
                                   const int32_t* cmin, const uint8_t* fbits, const uint16_t* foff, uint32_t* ukeys,
                                   cudaStream_t st) {
    if (maxB <= 0) return cudaSuccess;
    k_pack_from_codes<<<dim3(blocks_for(maxB), L), NT, 0, st>>>(boff, codes, M, KW, cmin, fbits, foff, ukeys);
    return cudaGetLastError();
}

cudaError_t launch_random_projection(float* A, float* u, int64_t nA, int64_t nu, unsigned long long seed,
                                     cudaStream_t st) {
    const int64_t n = std::max(nA, nu);
    if (n <= 0) return cudaSuccess;
    k_random<<<blocks_for(n), NT, 0, st>>>(A, u, nA, nu, seed);
    return cudaGetLastError();
}

}  // namespace culsh
