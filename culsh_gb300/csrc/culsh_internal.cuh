// Internal declarations shared by the CUDA translation units of libculsh.
//
// Device data model of one index (all tables stacked, one allocation each):
//   X        [N][D]  f32    dataset, point-contiguous (the reference's D x N column-major)
//   A        [L*M][D] f32   projection columns; column (l,m) = A[l][m*D .. m*D+D)
//   b        [L*M]   f32
//   cmin/cmax[L*M]   i32    per (table, column) code range
//   fbits/foff[L*M]         bit width / bit offset of each column's field in the packed key
//   ids      [L][N]  u32    point ids sorted by (code row, id): the reference's totalIndices
//   boff     [L+1]   u64    bucket offsets: buckets of table l are [boff[l], boff[l+1])
//   starts/sizes [sum B]    bucket start (within the table's ids) and size
//   ukeys    [sum B][KW]    packed key of each bucket (column 0 in the most significant bits)
//   hslots   [sum H]  u64   bucketized open-addressing hash in 32-byte groups (one
//                           DRAM sector, kGroupWords u64): word 0 holds four 16-bit
//                           fingerprints (0xFFFF = empty), words 1-2 the four 32-bit
//                           bucket indices; probing visits a group's slots in order,
//                           then the next group
//   hoff     [L+1]   u64    word offsets of each table's groups
//   hmask    [L]     u32    power-of-two group count - 1
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>
#include <cuda_runtime.h>

struct culsh_index;

namespace culsh {

// Makes an index and its dataset device-resident (capi.cu).
int index_make_resident(culsh_index* ix);

constexpr int kMaxM = 64;     // projection columns per table
constexpr int kMaxKW = 8;     // packed key words (256 bits)
constexpr int kMaxT = 256;    // probes per table
constexpr int kMaxK = 2048;   // neighbours per query
constexpr unsigned long long kEmptySlot = ~0ull;
constexpr int kGroupSlots = 4;   // hash slots per 32-byte group
constexpr int kGroupWords = 4;   // u64 words per group
constexpr uint32_t kEmptyFp = 0xFFFFu;

// 16-bit slot fingerprint from the top bits of a key hash (never the empty mark).
__host__ __device__ __forceinline__ uint32_t slot_fp(uint64_t hh) {
    const uint32_t f = (uint32_t)(hh >> 48);
    return f == kEmptyFp ? kEmptyFp - 1 : f;
}

// Device error flags (bit values OR-ed into an int in device memory).
enum DevErr : int {
    kErrNonFinite = 1,     // projection produced NaN/Inf
    kErrCodeRange = 2,     // |code| >= 2^31
    kErrSpin = 4,          // a bounded wait gave up
    kErrHashFull = 8,      // hash insert ran out of probes
    kErrNotIntegral = 16,  // a loaded bucket code is not an integer
};

// splitmix64 finalizer (Steele, Lea, Flood, OOPSLA 2014; public domain).
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__host__ __device__ __forceinline__ uint32_t mix32(uint32_t h) { return (uint32_t)mix64(h); }

constexpr uint64_t kHashSeed = 0x2545f4914f6cdd1dull;

// Lookup hash of a bucket key, additive in its fields: h = sum_m f_m * R_c
// (mod 2^64) over the fields f_m = code_m - cmin_m of table l, with R_c an
// odd 64-bit multiplier per column c = l * M + m, then one mix. A multiprobe
// key differs from its home key by +-1 in some fields, so its hash is the
// home sum +- R_c before the mix. Equal keys hash equally; a lookup verifies
// the stored key on every fingerprint match, so collisions cost time only.
__host__ __device__ __forceinline__ uint64_t field_mult(int c) {
    return mix64(kHashSeed ^ (0x9E3779B97F4A7C15ull * (uint64_t)(c + 1))) | 1ull;
}
__host__ __device__ __forceinline__ uint64_t hash_finish(uint64_t h) { return mix64(h ^ kHashSeed); }

// Key filter beside each table's hash (a blocked Bloom filter, two bits in
// one 32-bit word per two groups, 8 to 16 bits per key). The word is that of
// the key's home group, so that a part of a table and its filter are built
// together; the bits are independent of the group (low 32 bits), one of them
// is part of the fingerprint (top 16 bits, the same for the two hashes that
// slot_fp makes equal). A key that is in the table always finds both set.
__host__ __device__ __forceinline__ uint32_t filter_word(uint64_t hh) { return (uint32_t)hh >> 1; }
__host__ __device__ __forceinline__ uint32_t filter_bits(uint64_t hh) {
    return (1u << ((uint32_t)(hh >> 43) & 31u)) | (1u << ((uint32_t)(hh >> 53) & 31u));
}

// Place a field of `bits` bits (<= 32) at bit offset `off` of a little-endian
// multi-word key.
__host__ __device__ __forceinline__ void key_put(uint32_t* key, int off, int bits, uint32_t val) {
    const int w = off >> 5, s = off & 31;
    key[w] |= val << s;
    if (s != 0 && s + bits > 32) key[w + 1] |= val >> (32 - s);
}

__host__ __device__ __forceinline__ uint32_t key_get(const uint32_t* key, int off, int bits) {
    if (bits == 0) return 0;
    const int w = off >> 5, s = off & 31;
    uint64_t v = key[w] >> s;
    if (s != 0 && s + bits > 32) v |= (uint64_t)key[w + 1] << (32 - s);
    return bits == 32 ? (uint32_t)v : (uint32_t)(v & ((1ull << bits) - 1));
}

// Per-table key layout and lookup structures (device pointers).
struct LookupView {
    int L, M, KW;
    const int32_t* cmin;
    const int32_t* cmax;
    const uint8_t* fbits;
    const uint16_t* foff;
    const uint64_t* boff;
    const uint32_t* starts;
    const uint32_t* sizes;
    const uint32_t* ukeys;
    const unsigned long long* hslots;
    const uint64_t* hoff;
    const uint32_t* hmask;
    const unsigned long long* funit;   // [L*M][2]: 2^foff as (low, high) 64-bit words
    const unsigned long long* rmul;    // [L*M]: field multipliers of the lookup hash
    const uint32_t* filt;              // key filters, table l at words [fl_off[l], fl_off[l+1])
    const uint64_t* fl_off;
    const uint32_t* fl_mask;           // [L]: words in table l's filter - 1 (half its groups, at least one)
};

// ---------------------------------------------------------------------------
// Launchers (each returns cudaGetLastError() after the launch).

// Canonical FP32 projection of n_pts points onto the LM stacked columns.
// codes != nullptr: floored codes [LM][n_pts] + per-block min/max partials
// [grid_x][LM]; vals != nullptr: unfloored values [LM][n_pts].
// tile picks the query-value tiling (0: 64x128, 1: 32x128, 2: 128x64 points x columns).
// Word arrays a kernel zeroes on the way (grid-stride, every block takes
// part): the search's first kernel clears the counters the later ones
// accumulate into, instead of two memset nodes in the graph.
struct ZeroWords {
    unsigned long long* a = nullptr;
    int64_t na = 0;
    unsigned long long* b = nullptr;
    int64_t nb = 0;
    __device__ __forceinline__ void clear(int tid) const {
        if (!na && !nb) return;
        const int64_t nthreads = (int64_t)gridDim.x * gridDim.y * blockDim.x;
        const int64_t g = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + tid;
        for (int64_t i = g; i < na; i += nthreads) a[i] = 0ull;
        for (int64_t i = g; i < nb; i += nthreads) b[i] = 0ull;
    }
};

// AT: the projection matrix transposed, D rows of lmp floats (lmp = LM rounded
// up to a multiple of 4, columns past LM zero, 16-byte aligned).
cudaError_t launch_project_fp32(const float* X, int64_t n_pts, int D, const float* AT, int lmp, const float* b,
                                int LM, float W, int32_t* codes, float* vals, int32_t* pmin, int32_t* pmax, int* err,
                                cudaStream_t st, int tile = 0, ZeroWords zw = ZeroWords{}, float* xcopy = nullptr);
int project_grid_x(int64_t n_pts);
// The kernel that the xcopy form launches for n_pts rows, for finding its node
// in a captured graph, and its number of parameters (the first is the rows it
// reads).
const void* project_copy_kernel(int64_t n_pts, int D, int LM);
constexpr int kProjectArgs = 15;
// n floats, 16-byte aligned source and destination (src may be host memory
// the device reads directly).
cudaError_t launch_copy_f32(const float* src, float* dst, int64_t n, cudaStream_t st);
cudaError_t launch_minmax_reduce(const int32_t* pmin, const int32_t* pmax, int nparts, int LM, int32_t* cmin,
                                 int32_t* cmax, cudaStream_t st);

// Tensor-core (tcgen05) projection for index builds: plan, fp16 split of X,
// the GEMM with the proven-code epilogue, and the canonical recomputation of
// the codes its error bound could not prove.
// Scales and properties of a projection's operands (device).
struct ProjectState {
    uint32_t amax_x, amax_a;   // largest magnitudes (float bits): X's sample, A
    float sx, sa;              // power-of-two scales
    int flags;                 // see k_split_rows
};
struct TcPlan {
    bool ok;
    int Dp, blk, LMp, ntiles, grid;   // columns of one launch, of all launches
    uint32_t b_bytes, x_bytes;
    int stages[2];        // X-tile ring depth without / with the low fp16 part
    size_t smem[2];
};
TcPlan tc_plan(int64_t N, int D, int LM, int num_sms, int max_smem);
// Streaming form for projections whose matrix does not fit shared memory:
// column blocks of blk[need_lo] per launch, any Dp.
struct TcStreamPlan {
    bool ok;
    int Dp, LMp, ntiles, grid;
    int blk[2], stages[2];
    size_t smem[2];
};
TcStreamPlan tc_plan_stream(int64_t N, int D, int LM, int num_sms, int max_smem);
cudaError_t launch_project_tc_stream(const TcStreamPlan& p, int need_lo, int64_t N, int D, int LM, const void* xh,
                                     const void* xl, const void* ah, const void* al, const float* b,
                                     const float* anorm, const float* xnorm, const ProjectState* ps, float W, float kappa,
                                     int32_t* codes, int32_t* pmin, int32_t* pmax, unsigned long long* relist,
                                     unsigned long long relist_cap, unsigned int* relist_cnt, int* err,
                                     cudaStream_t st);
// Norms of A's columns and of ns rows of X, and both scales; fp16 parts of A and
// of X (xl null: the high part only; rescale: from X's own maximum).
cudaError_t launch_project_sample(const float* X, int64_t N, int D, int ns, const float* A, int LM, float slope, float* xs,
                                  float* anorm, ProjectState* ps, cudaStream_t st);
cudaError_t launch_split_a(const float* A, int LM, int LMp, int D, int Dp, float kappa, float slope, void* ah, void* al, float* anorm,
                           const ProjectState* ps, cudaStream_t st);
cudaError_t launch_split_rows(const float* X, int64_t N, int D, int Dp, float kappa, float slope, void* xh, void* xl, float* xnorm,
                              ProjectState* ps, bool rescale, cudaStream_t st);
cudaError_t launch_project_tc(const TcPlan& p, int need_lo, int64_t N, int D, int LM, const void* xh, const void* xl,
                              const void* ah, const void* al, const float* b, const float* anorm, const float* xnorm,
                              const ProjectState* ps, float W, float kappa, int32_t* codes, int32_t* pmin, int32_t* pmax,
                              unsigned long long* relist, unsigned long long relist_cap, unsigned int* relist_cnt,
                              int* err, cudaStream_t st);
cudaError_t launch_tc_recompute(const float* X, int64_t N, int D, int LM, const float* A, const float* b, float W,
                                const unsigned long long* list, unsigned long long cap, const unsigned int* cnt,
                                int regions, int32_t* codes, int32_t* cmin, int32_t* cmax, int* err, cudaStream_t st);

// Key packing from int codes [LM][N] into SoA keys [KW][L*N] and identity values;
// with low (KW 2 to 4): the top word into keys [L*N], the lower words into rows
// of lw words (low_row_words).
cudaError_t launch_pack_keys(const int32_t* codes, int64_t N, int L, int M, int KW, const int32_t* cmin,
                             const uint8_t* fbits, const uint16_t* foff, uint32_t* keys, uint32_t* vals,
                             uint32_t* low, int lw, cudaStream_t st);

// Onesweep segmented LSD radix sort of L segments of N (key, value) pairs.
// Sorts bits [0, 8*passes) of the KW-word keys. Buffers are ping-ponged; on
// return *result_in_alt tells whether the sorted data sits in the alt buffers.
struct SortBuffers {
    uint32_t* keys[2];   // [KW][L*N] each
    uint32_t* vals[2];   // [L*N] each
    uint32_t* hist;      // [L][passes][256]
    uint32_t* base;      // [L][passes][256]
    uint32_t* status;    // [L*tiles][256] + counter
    int* err;
};
size_t sort_status_words(int64_t N, int L);
// Digits below first_pass are zero in every key and get no pass.
cudaError_t run_segmented_sort(SortBuffers& sb, int64_t N, int L, int KW, int passes, int first_pass,
                               bool* result_in_alt, cudaStream_t st);

// Top-word-first ordering (sort.cu): after the digit passes over the top key
// word, find the runs of equal top words and order each run by (lower words,
// id).
struct RunLists {
    unsigned long long* tpos;   // runs of 3..8: first sorted position (table * N + i)
    uint32_t* tlen;
    unsigned int tcap;
    unsigned long long* spos;   // runs of 9..32
    uint32_t* slen;
    unsigned int scap;
    unsigned long long* lpos;   // runs of 33..2,048 (kRunMax)
    uint32_t* llen;
    unsigned int lcap;
    uint32_t* same;             // bit per sorted position: same key as the one before (launch_rl_count's flags)
    unsigned int* cnt;          // [4]: tiny, small and large runs; overflow flags (1 run too long, 2 list full)
};
cudaError_t launch_run_find(const uint32_t* top, int64_t N, int L, int KW, const uint32_t* low, uint32_t* ids,
                            const RunLists& rl, cudaStream_t st);
cudaError_t launch_run_sorts(const RunLists& rl, int64_t N, int L, int KW, const uint32_t* low, uint32_t* ids,
                             cudaStream_t st);

// Sorted keys of all tables: KW arrays of L*N words, or (low != nullptr) the
// sorted top words and the lower words by point, in rows of lw words.
struct SortedKeys {
    const uint32_t* keys;
    const uint32_t* low;
    const uint32_t* ids;   // [L*N] sorted ids
    int lw;
};
constexpr int low_row_words(int KW) { return KW == 2 ? 1 : KW == 3 ? 2 : 4; }

// Run-length bucketing of sorted keys. Two phases: count (boundary flags, one
// word per 32 positions of 4,096-position tiles; per table bucket totals,
// written to nb[L]) and write (starts, ukeys).
cudaError_t launch_rl_count(const SortedKeys& keys, int64_t N, int L, int KW, uint32_t* tile_cnt, uint32_t* tile_off,
                            uint32_t* flags, uint32_t* nb, cudaStream_t st);
cudaError_t launch_rl_write(const SortedKeys& keys, int64_t N, int L, int KW, const uint32_t* flags,
                            const uint32_t* tile_off, const uint64_t* boff, uint32_t* starts, uint32_t* ukeys,
                            cudaStream_t st);
// Hash tables and filters over the unique keys; with sizes set also the bucket
// sizes and the largest (max_size zeroed by the caller).
struct HashBuild {
    const uint64_t* boff;
    const uint32_t* ukeys;
    int L, M, KW;
    int64_t maxB;                 // most buckets of a table
    uint32_t max_groups;          // most groups of a table
    const uint16_t* foff;
    const uint8_t* fbits;
    const unsigned long long* rmul;
    const uint64_t* hoff;
    const uint32_t* hmask;
    unsigned long long* hslots;
    uint32_t* filt;
    const uint64_t* fl_off;
    const uint32_t* fl_mask;
    const uint32_t* starts;       // with sizes: a build's bucket starts, points per table
    int64_t N;
    uint32_t* sizes;
    uint32_t* max_size;
    int* err;
    // Form by parts: records [L][parts of the largest table][kHashPartCap], their
    // counts, keys that fit no part's records or slots.
    unsigned long long* rec;
    uint32_t* part_cnt;           // [L][parts], then the spill count
    uint2* spill;                 // (table, bucket)
    uint32_t spill_cap;
    uint32_t part_cap;            // records a part takes, at most kHashPartCap
};
constexpr uint32_t kHashPartGroups = 2048;   // groups built together in shared memory
constexpr uint32_t kHashPartCap = 4672;      // a part's records: 4,096 expected at most, 9 deviations more
constexpr uint32_t kHashMaxParts = 4096;
// Key by key in place (hslots all ones, filt zero), or by parts (any contents).
cudaError_t launch_hash_build(const HashBuild& h, cudaStream_t st);
cudaError_t launch_hash_build_parts(const HashBuild& h, cudaStream_t st);
// Bucket codes [M][B_l] per table (float, the reference's layout) decoded from ukeys.
cudaError_t launch_decode_codes(const uint64_t* boff, const uint32_t* ukeys, int L, int M, int KW, int64_t maxB,
                                const int32_t* cmin, const uint8_t* fbits, const uint16_t* foff, float* codes,
                                cudaStream_t st);
// From loaded float bucket codes: per (l,m) min/max + integrality check, then ukeys.
cudaError_t launch_codes_minmax(const uint64_t* boff, const float* codes, int L, int M, int64_t maxB,
                                int32_t* cmin, int32_t* cmax, int* err, cudaStream_t st);
cudaError_t launch_pack_from_codes(const uint64_t* boff, const float* codes, int L, int M, int KW, int64_t maxB,
                                   const int32_t* cmin, const uint8_t* fbits, const uint16_t* foff, uint32_t* ukeys,
                                   cudaStream_t st);

// Random projection (seeded counter-based generator): A ~ N(0,1), u ~ U(0,1].
cudaError_t launch_random_projection(float* A, float* u, int64_t nA, int64_t nu, unsigned long long seed,
                                     cudaStream_t st);

// Query side.
struct ProbeArgs {
    const float* vals;         // [L*M][Q] unfloored projections
    int Q, T;
    LookupView lv;
    int32_t* qbuckets;         // [L][Q*T]
    unsigned long long* cnu;   // [Q] non-unique candidate counts (accumulated)
    int small_codes;           // every |cmin|, |cmax| < 2^24 - 2 (set by the host)
    int auto_form;             // no probe form was set by the caller: small batches may take a warp per pair
    int pch;                   // fast kernel: probes whose group loads overlap (1, 2, 4)
    // Split lookups (M <= 16, fast kernel). split = 1: the enumeration kernel
    // stores each valid probe's finished hash and mask and marks its query
    // bucket -2; k_probe_resolve then checks the key filter and walks the
    // hash. split = 2: the enumeration kernel stores them and looks its
    // pair's probes up itself, behind the filter, at its end.
    int split;
    unsigned long long* ph;    // [L][T][Q] finished hash of each pending probe
    uint32_t* pmask;           // [L][T][Q] its mask over the sorted deltas
    uint4* pctx;               // [L*Q][3] home key (128 bits), sorted deltas (32 bytes)
};
cudaError_t launch_probe(const ProbeArgs& a, cudaStream_t st);
int probe_launches(const ProbeArgs& a);   // kernels launch_probe launches

struct CandArgs {
    const float* X;
    int64_t N;
    int D, L, T, Q, K;
    const float* queries;              // [Q][D]
    const int32_t* qbuckets;           // [L][Q*T]
    const uint64_t* boff;
    const uint32_t* starts;
    const uint32_t* sizes;
    const uint32_t* ids;               // [L][N]
    const unsigned long long* cnu;     // [Q]
    int32_t* out_ids;                  // [Q][K]
    float* out_d;                      // [Q][K]
    unsigned long long* cu;            // [Q] unique counts
    unsigned long long* totals;        // [2]: sum unique, sum non-unique
    uint32_t* arena;                   // overflow hash sets for large candidate sets
    unsigned long long arena_words;
    unsigned long long* arena_top;
    int* deferred;                     // [Q] list of queries that did not fit the arena
    unsigned int* n_deferred;
    const int* qlist;                  // optional subset of queries (nullptr = all)
    int nq;
};
// Work-stealing form of the candidate stage (candidates.cu): queries split
// into id-partition items, claimed by a persistent grid.
// How the work-stealing kernel reads candidate rows: FP32 rows straight from
// global memory, BF16 copies with an FP32 recheck, FP32 rows staged in shared
// memory by bulk copies (sets of 4,096 slots).
enum class WsForm : int { direct = 0, bf16 = 1, staged = 2 };

struct WsArgs {
    const float* X;
    int64_t N;
    int D, L, T, Q, K;
    const float* queries;              // [Q][D]
    const int32_t* qbuckets;           // [L][Q*T]
    const uint64_t* boff;
    const uint32_t* starts;
    const uint32_t* sizes;
    const uint32_t* ids;               // [L][N]
    const unsigned long long* cnu;     // [Q]
    int32_t* out_ids;                  // [Q][K]
    float* out_d;                      // [Q][K]
    unsigned long long* cu;            // [Q] unique counts
    unsigned long long* totals;        // [2]: sum unique, sum non-unique
    int pmax;                          // partitions per query, at most 64
    unsigned long long chunk;          // non-unique candidates per partition
    unsigned long long whole;          // ... up to which a query is one item whatever chunk says
    int* q_items;                      // [Q] partitions of each query
    int* q_off;                        // [Q] first item of each query
    unsigned int* q_done;              // [Q] partitions finished
    int* item_q;                       // [item_cap]
    uint8_t* item_p;                   // [item_cap]
    int* part_n;                       // [item_cap] partial list lengths
    float* part_d;                     // [item_cap][K]
    uint32_t* part_i;                  // [item_cap][K]
    unsigned int item_cap;
    unsigned int* n_items;
    unsigned int* next_item;           // work-stealing counter, zero before the launch
    unsigned int* overflow;            // nonzero: rerun with the per-query kernel
    // Queries of 1 .. small_max non-unique candidates (0: none), one warp each
    uint32_t small_max;
    int* small_q;                      // [Q]
    unsigned int* n_small;
    int wt;                            // threads per item CTA: 64, 128 or 256
    int slots;                         // shared hash-set slots per item: 4096 or 8192
    // BF16 form: approximate distances from xb, certified FP32 rerank
    WsForm form;
    const uint16_t* xb;                // [N][D] bf16 copy of X
    const uint8_t* xflag;              // [N] 1 exact in bf16, 2 always re-check, 0 bound applies
    float e_c1, e_c2;                  // error-bound factors (rounded up)
    unsigned long long* rechecked;     // candidates whose FP32 row pass 2 re-read
    // Dense form: queries with at least dense_min non-unique candidates
    unsigned long long dense_min;      // ~0ull: never
    int* dense_q;                      // [Q] queries routed to the bitmap kernel
    unsigned int* n_dense;
    unsigned int* dense_next;          // claim counter of the bitmap kernel
    // Locality order (tuned): queries planned in the order of their home
    // bucket in table 0 (launch_order_queries), so that items of queries
    // with shared candidates run close together and share rows in L2.
    uint32_t* order;                   // [Q] queries in that order; nullptr: index order
    uint32_t* order_bins;              // [kOrderBins + 1] counting-sort bins
    // Bucket rows (tensor-core path): the index's largest buckets as N-bit
    // rows, ORed into a dense query's membership row instead of setting the
    // bits of their ids one by one. big_gi holds their global bucket numbers
    // (boff[l] + j) in ascending order; every bucket of big_min ids or more
    // has a row. nbig == 0: none.
    const uint64_t* big_gi;
    const uint32_t* big_rows;          // [nbig][nwp]
    int nbig;
    uint32_t big_min;
    // Bank lists (tensor-core path, one membership segment): the ids of every
    // bucket of bank_min ids or more again, arranged for the membership kernel
    // (k_bank_fill). bank_meta[g] of global bucket g: (groups of 128 entries,
    // tail ids). nullptr: none.
    const uint16_t* bank;
    const uint32_t* bank_tail;
    const uint2* bank_meta;
    uint32_t bank_min;
};
constexpr uint32_t kBankMin = 512;            // smallest bucket that has a bank list
constexpr int64_t kBankMaxN = (int64_t(1) << 21) - 1024;   // 11 bits of word row (one past the bitmap), 5 of bit
constexpr uint32_t kSmallMax = 32;     // candidates a warp's lanes hold
constexpr int kSmallMaxD = 1024;       // dimensions whose query rows leave several blocks resident
cudaError_t launch_candidates_small(const WsArgs& a, int sms, cudaStream_t st);
constexpr int kOrderBins = 4096;
cudaError_t launch_order_queries(const WsArgs& a, cudaStream_t st);   // 3 kernels + 1 memset
size_t dense_smem_bytes(int64_t N, int D, int K);
cudaError_t launch_candidates_dense(const WsArgs& a, int grid, cudaStream_t st);
size_t ws_smem_bytes(int D, int K, int wt, WsForm form, int slots);
int ws_blocks_per_sm(int D, int K, int wt, WsForm form, int slots);
cudaError_t launch_bf16_rows(const float* X, int64_t N, int D, uint16_t* xb, uint8_t* flag, cudaStream_t st);
cudaError_t launch_plan_items(const WsArgs& a, cudaStream_t st);
// Bucket rows: the global numbers and sizes of the buckets of at least
// big_min ids (at most cap, in no order; *cnt counts them), then their rows
// (rows zeroed beforehand; tl[r] is bucket r's table).
cudaError_t launch_big_find(const uint32_t* sizes, uint64_t totB, uint32_t big_min, uint64_t* gi, uint32_t* sz,
                            unsigned int* cnt, unsigned int cap, cudaStream_t st);
cudaError_t launch_big_fill(const uint64_t* gi, const int32_t* tl, int nbig, const uint32_t* starts,
                            const uint32_t* sizes, const uint32_t* ids, int64_t N, uint32_t* rows, int nwp,
                            cudaStream_t st);
// Bank lists of the n buckets gi (any order): see k_bank_fill.
cudaError_t launch_bank_fill(const uint64_t* gi, const unsigned int* n, unsigned int cap, const uint64_t* boff, int L,
                             const uint32_t* starts, const uint32_t* sizes, const uint32_t* ids, int64_t N,
                             uint16_t* bank, uint32_t* tail, uint2* meta, cudaStream_t st);
cudaError_t launch_candidates_ws(const WsArgs& a, int grid, cudaStream_t st);

// ---------------------------------------------------------------------------
// Tensor-core k-NN over candidate membership rows (knn_tc.cu): the dense
// queries' candidate distances and top-K as a masked GEMM.

// Properties of the dataset's values, accumulated by k_knn_scan and
// k_knn_rows. Zero is the empty state.
enum KnnFlags : int {
    kKnnNotSmallInt = 2,   // some value is not an integer of magnitude <= 256
    kKnnNonFinite = 4,
};
struct KnnState {
    int flags;
    int mneg;        // max over the small-integer values v of 257 - v (0: none)
    int mpos;        // max over them of v + 257
    uint32_t amax;   // largest magnitude (float bits)
    uint32_t rho;    // largest relative fp16 residual of a row (float bits)
};
// A dense query's key multipliers and error terms (knn_tc.cu).
enum KnnQueryFlags : int {
    kKnnExact = 1,   // small integers: keys are exact
    kKnnUnfit = 2,   // magnitudes outside the tensor-core path: scanned exactly
};
struct KnnQuery {
    float m_lo, m_up;     // of the lower- and upper-bound keys
    float sq;             // |q|^2
    float kappa, slack;
    int flags;
};
constexpr int kMaxKnnK = 256;           // neighbours the tensor-core path serves
constexpr int kMaxKnnD = 2048;          // dimensions
constexpr int kKnnTileQ = 256;          // queries per tensor-core tile
constexpr int kKnnMaxSurvivors = 4096;  // candidates of a query the merge takes
constexpr int kKnnMaxChosen = 1024;     // of those, distances it computes
// Magnitudes (largest of a row or of the dataset) outside which squares could
// leave the float range.
constexpr float kKnnMaxValue = 1e17f, kKnnMinValue = 1e-12f;

// Everything the k-NN kernels of one search read and write.
struct KnnSearch {
    int N, D, Dp, K;
    int nd, Qcap;                      // dense queries; rows of the query buffers (nd rounded up to kKnnTileQ)
    int grid;                          // persistent CTAs of the tensor-core kernels
    int ops;                           // operand ring stages
    size_t smem;                       // dynamic shared memory of the tensor-core kernels
    int nwp;                           // membership words per query row (a multiple of 4)
    // sample pass: every f-th point (0: none) of nseg segments of seg points,
    // in s32 chunks of 32 each; chunk c of segment g holds the points
    // g seg + (i s32 + c) f, i < 32
    int f, nseg, seg, s32;
    int nws;                           // sample membership words per query row
    float gamma;
    // dataset side (per index)
    const void* xh;                    // [N][Dp] fp16, scaled
    const float* w;                    // [N padded to 256]: |x|^2, FLT_MAX past N
    const KnnState* dstate;
    const float* X;                    // [N][D] f32 (exact distances)
    // query side (per search)
    const float* queries;              // [Q][D] f32
    const int* dense_q;                // dense list (query ids)
    void* qh;                          // [Qcap][Dp] fp16, dense-list order
    KnnQuery* qinfo;                   // [Qcap]
    float* qlim;                       // [Qcap]
    float* w_sample;                   // [nws * 32]
    float* smin;                       // [Qcap][nws] chunk minima
    const uint32_t* bm;                // [Qcap][nwp] membership rows (k_cand_bitmap)
    uint32_t* bm_sample;               // [Qcap][nws] their sample points
    uint2* part;                       // survivor lists, list_cap entries each
    int* part_n;
    int list_cap;
    int32_t* out_ids;
    float* out_d;
    int* fallback;                     // [Qcap] dense positions to scan exactly
    unsigned int* n_fallback;
    int* err;
};
// Buffer sizes of one search (elements).
size_t knn_part_entries(const KnnSearch& k);   // part entries
size_t knn_part_lists(const KnnSearch& k);     // part_n entries
// Plans shared memory, sample and list sizes for N, D, K, Qcap and grid; false
// when the tensor-core path does not serve them. bitmap_smem: shared memory
// the membership kernel may use for its bitmap.
bool knn_plan(KnnSearch& k, int max_smem, size_t bitmap_smem);
// Relative error terms beside the operand residuals (see knn_tc.cu).
float knn_gamma(int D);
// Dataset rows: fp16 operand, norms, state (once per index).
cudaError_t launch_knn_rows_dataset(const float* X, int64_t N, int D, int Dp, void* xh, float* w, int64_t pad,
                                    KnnState* st, cudaStream_t s);
// Query rows, tensor-core passes and merge of one search.
cudaError_t launch_knn_search(const KnnSearch& k, cudaStream_t s);
int knn_launches(const KnnSearch& k);
// Membership rows of the dense queries, and the exact scan of the queries the
// merge could not finish (candidates.cu).
size_t bitmap_smem(int max_smem);   // bytes of bits a membership block can hold
cudaError_t launch_cand_bitmap(const WsArgs& a, const KnnSearch& k, uint32_t* bm, int grid, cudaStream_t st);
cudaError_t launch_knn_scan_rows(const KnnSearch& k, int grid, cudaStream_t st);
size_t knn_scan_smem(int D, int K);

// Opts `func` into `dyn` bytes of dynamic shared memory: always, whatever the
// size, since the 48 KB that need no opt-in include the kernel's static part
// (15 KB of k_cand_bitmap, whose launches of 33 to 36 KB more had been refused).
// The opted-in size only grows (`cap` records it per kernel), so a smaller
// configuration launched later stays valid.
template <class F>
cudaError_t opt_in_smem(F* func, size_t dyn, std::atomic<size_t>& cap) {
    if (dyn <= cap.load()) return cudaSuccess;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (dyn <= cap.load()) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e == cudaSuccess) cap = dyn;
    return e;
}

// Process-wide lock held while a search plans (and grows) its buffers and
// captures its graph: no thread frees device memory while another captures.
std::mutex& alloc_capture_mutex();
// culsh_search_estimate_bytes, with or without the tensor-core path's buffers.
long long search_estimate(const culsh_index* ix, int Q, int K, int T, bool tensor_cores);
// Sets the calling thread's culsh_last_error() message; returns code.
int set_last_error(int code, const char* msg);

int cand_smem_capacity();              // candidates handled in shared memory per query
cudaError_t launch_candidates(const CandArgs& a, cudaStream_t st);
size_t cand_arena_words(unsigned long long nonunique);

}  // namespace culsh
