// COO -> CSR / CSC conversion with optional fused gcn_norm, for sm_100a.
//
// Replaces the reference's host-side, single-thread counting sorts
// (ops/cpp/cootocsr_op.cc:24-57, ops/cpp/cootocsc_op.cc:23-53) and the tensor-level
// gcn_norm / add_remaining_self_loops (nn/conv/gcn_conv.py:18-37, utils/loop.py:120-134).
//
// Layout contract (bit-exact with the reference): entry i of the COO list lands at
// off[key_i] + #{j < i : key_j == key_i}, i.e. a STABLE sort on the row key; with gcn_norm the
// list is the input with (v,v) entries removed followed by one loop per node in node order.
//
// Method: stable least-significant-digit radix sort, 8 bits per pass, ceil(bits(n)/8) passes,
// carrying (key, other index, weight).  Each pass = per-tile digit histogram, one device-wide
// exclusive scan of the [tile][digit] count matrix in digit-major order, and a stable scatter: ranks inside a tile come from
// per-digit masks of the warp (votes, or matches on a list in runs) in element order, elements are staged in shared memory in digit order and
// written out in coalesced runs.  The first pass reads the caller's COO directly (self-loop
// removal and the appended loops are folded into it: removed entries are simply never counted),
// the last pass writes the caller's output arrays.  Offsets are found from the sorted keys by
// boundary detection; nothing uses floating-point atomics, so results are run-to-run identical.
// About 20 bytes per entry and pass (4 histogram read, 8 read, 8 write; 12 more with weights to carry).  The scatter
// is bound by the SM, not by DRAM: 37 shared-memory and load/store wavefronts and some 60 integer instructions per
// 32 entries (ranks, staging, write-out) are 1.65 ms of a 285 M-entry pass against 0.7 ms for its bytes.
#include "common.cuh"
#include "scan.cuh"

namespace jg {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kRadix = 256;
// Entries per thread of a tile.  Sixteen halve the count matrix and its scans and lengthen the write runs (285 M
// unit-weight entries, three passes, two formats: 14.9 against 15.9 ms), but a third array to carry spills
// (30 M weighted entries: 3.1 against 2.6 ms), and a list of fewer than some 2 M entries would leave SMs
// without a tile.
constexpr int kItemsFew = 8, kItemsMany = 16;
constexpr int kMatchRuns = 8;      // runs of equal digits in 32 elements up to which a match mask beats the votes
constexpr int64_t kManyEntries = (int64_t)1 << 21;
static inline int sort_items(int64_t count, bool carry_w) { return !carry_w && count >= kManyEntries ? kItemsMany : kItemsFew; }
static inline int64_t sort_tiles(int64_t count, int items) {
    return (count + (int64_t)kSortThreads * items - 1) / ((int64_t)kSortThreads * items);
}

// ------------------------------------------------------------------------------- digit-major scan
// The per-tile digit counts live as matrix[tile][digit] (rows of 256 counts, written and read
// coalesced).  The scatter needs, for every (digit, tile), the number of entries with a smaller
// digit anywhere plus the entries with the same digit in earlier tiles: an exclusive scan in
// digit-major order.  It is done column-wise, thread d walking column d, so every access is a
// coalesced row: chunk sums, one block that scans chunks and digits, then a walk down each chunk.
constexpr int kChunkTiles = 128;

__global__ void __launch_bounds__(kRadix) colscan_chunk_sums(const int* __restrict__ matrix, int64_t n_tiles,
                                                             int* __restrict__ chunk_sums) {
    const int64_t t0 = (int64_t)blockIdx.x * kChunkTiles;
    const int64_t t1 = t0 + kChunkTiles < n_tiles ? t0 + kChunkTiles : n_tiles;
    int sum = 0;
    for (int64_t t = t0; t < t1; t++) sum += matrix[t * kRadix + threadIdx.x];
    chunk_sums[(int64_t)blockIdx.x * kRadix + threadIdx.x] = sum;
}

// `total` (or null) receives the number of entries counted.
__global__ void __launch_bounds__(kRadix) colscan_chunks(int* __restrict__ chunk_sums, int64_t n_chunks,
                                                         unsigned long long* __restrict__ total) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    int run = 0;
    for (int64_t c = 0; c < n_chunks; c++) {          // exclusive prefix of this digit's chunk sums
        const int v = chunk_sums[c * kRadix + threadIdx.x];
        chunk_sums[c * kRadix + threadIdx.x] = run;
        run += v;
    }
    const int base = block_exclusive_scan(run, &s_total, s_warp);   // entries with a smaller digit
    if (total && threadIdx.x == 0) *total = (unsigned long long)s_total;
    for (int64_t c = 0; c < n_chunks; c++) chunk_sums[c * kRadix + threadIdx.x] += base;
}

__global__ void __launch_bounds__(kRadix) colscan_apply(int* __restrict__ matrix, int64_t n_tiles,
                                                        const int* __restrict__ chunk_sums) {
    const int64_t t0 = (int64_t)blockIdx.x * kChunkTiles;
    const int64_t t1 = t0 + kChunkTiles < n_tiles ? t0 + kChunkTiles : n_tiles;
    int run = chunk_sums[(int64_t)blockIdx.x * kRadix + threadIdx.x];
    for (int64_t t = t0; t < t1; t++) {
        const int v = matrix[t * kRadix + threadIdx.x];
        matrix[t * kRadix + threadIdx.x] = run;
        run += v;
    }
}

// The same in one launch for a matrix of at most kChunkTiles rows.
__global__ void __launch_bounds__(kRadix) colscan_small(int* __restrict__ matrix, int n_tiles, unsigned long long* __restrict__ total) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    int sum = 0;
#pragma unroll 16
    for (int t = 0; t < n_tiles; t++) sum += matrix[t * kRadix + threadIdx.x];
    int run = block_exclusive_scan(sum, &s_total, s_warp);
    if (total && threadIdx.x == 0) *total = (unsigned long long)s_total;
    for (int t0 = 0; t0 < n_tiles; t0 += 16) {
        int v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = t0 + i < n_tiles ? matrix[(t0 + i) * kRadix + threadIdx.x] : 0;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (t0 + i < n_tiles) matrix[(t0 + i) * kRadix + threadIdx.x] = run;
            run += v[i];
        }
    }
}

// ------------------------------------------------------------------------------- sort passes
// Where a pass reads its elements from.
struct SortSrc {
    // mode 0: SoA buffers (key, idx, w) of `count` entries
    const int32_t* key;
    const int32_t* idx;
    const float* w;
    // mode 1: the caller's COO list (first pass)
    const int32_t* coo_src;
    const int32_t* coo_dst;
    const float* coo_w;       // null: unit weights
    const float* loop_w;      // weight of the appended loop of node v (null: 1)
    int64_t e0;               // input entries
    int64_t n_loops;          // appended loops (0 or n)
    int by;                   // 0: key = source, 1: key = destination
    int drop_loops;           // skip (v,v) input entries
    int mode;
    int64_t count;            // positions of the (virtual) list, an upper bound when dcount is set
    const unsigned long long* dcount;  // device-resident element count (mode 0 after a dropping pass)
};

struct Elem {
    int32_t key, idx;
    float w;
    bool valid;
};

// An element is fetched in two steps so that a tile's loads can all be issued before anything looks at a
// loaded value: load_raw only loads (what it returns is not inspected), finish_elem derives key, index and
// validity.  With the two fused, the self-loop test of the first pass (a == b) made every element wait for
// its own loads before the next element's were issued, and every element re-read the device-side count.
struct Raw {
    int32_t a, b;
    float w;
};

__device__ __forceinline__ int64_t list_count(const SortSrc& s) { return s.dcount ? (int64_t)*s.dcount : s.count; }

// MODE (0, 1, 2 as in SortSrc) is a template parameter: with the tests of the other modes compiled in, the first pass of a
// COO list carried their registers and branches (285 M entries: one more of them cost 0.75 ms a pass).
template <int MODE>
__device__ __forceinline__ Raw load_raw(const SortSrc& s, int64_t p, int64_t count) {
    Raw r;
    r.a = 0; r.b = 0; r.w = 1.f;
    if (p >= count) return r;
    if (MODE == 0) {
        r.a = s.key[p]; r.b = s.idx[p];
        if (s.w) r.w = s.w[p];
    } else if (MODE == 2) {
        // mirrored list: position 2i is edge i as given, 2i + 1 the same edge reversed
        const int64_t i = p >> 1;
        r.a = s.coo_src[i]; r.b = s.coo_dst[i];
        if (s.coo_w) r.w = s.coo_w[i];
    } else if (p < s.e0) {
        r.a = s.coo_src[p]; r.b = s.coo_dst[p];
        if (s.coo_w) r.w = s.coo_w[p];
    } else {
        const int32_t v = (int32_t)(p - s.e0);
        r.a = v; r.b = v;
        if (s.loop_w) r.w = s.loop_w[v];
    }
    return r;
}

template <int MODE>
__device__ __forceinline__ Elem finish_elem(const SortSrc& s, int64_t p, int64_t count, const Raw& r) {
    Elem e;
    e.valid = p < count;
    e.key = 0; e.idx = 0; e.w = r.w;
    if (!e.valid) { e.w = 0.f; return e; }
    if (MODE == 0) {
        e.key = r.a; e.idx = r.b;
    } else if (MODE == 2) {
        e.key = (p & 1) ? r.b : r.a;
        e.idx = (p & 1) ? r.a : r.b;
    } else {
        // an appended loop has a == b, so the swap does not matter to it
        e.key = s.by == 0 ? r.a : r.b;
        e.idx = s.by == 0 ? r.b : r.a;
        if (s.drop_loops && r.a == r.b && p < s.e0) e.valid = false;
    }
    return e;
}

// digit of an element for this pass: from the key, or (canonical order passes) from the index
__device__ __forceinline__ int digit_of(const Elem& e, int shift, int from_idx) {
    return ((from_idx ? e.idx : e.key) >> shift) & (kRadix - 1);
}

constexpr int kHistThreads = kSortThreads;
template <int MODE, int ITEMS>
__global__ void __launch_bounds__(kHistThreads) sort_hist_kernel(SortSrc s, int shift, int from_idx, int* __restrict__ matrix) {
    __shared__ int s_hist[kRadix];
    constexpr int kSortTile = kSortThreads * ITEMS;
    constexpr int kRounds = ITEMS;
    constexpr int kBatch = 8;
    static_assert(kRounds % kBatch == 0, "a tile is read in whole batches");
    s_hist[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    const int64_t count = list_count(s);
    if (MODE == 0) {
        // sorted-buffer passes: only the array the digit comes from is read (half the bytes of a full element)
        const int32_t* from = from_idx ? s.idx : s.key;
        if (base + kSortTile <= count && reinterpret_cast<uintptr_t>(from) % 16 == 0) {
            int4 v[kRounds / 4];
#pragma unroll
            for (int i = 0; i < kRounds / 4; i++) v[i] = reinterpret_cast<const int4*>(from + base)[i * kHistThreads + threadIdx.x];
#pragma unroll
            for (int i = 0; i < kRounds / 4; i++) {
                atomicAdd(&s_hist[(v[i].x >> shift) & (kRadix - 1)], 1);
                atomicAdd(&s_hist[(v[i].y >> shift) & (kRadix - 1)], 1);
                atomicAdd(&s_hist[(v[i].z >> shift) & (kRadix - 1)], 1);
                atomicAdd(&s_hist[(v[i].w >> shift) & (kRadix - 1)], 1);
            }
        } else {
            for (int i = 0; i < kRounds; i++) {
                const int64_t p = base + (int64_t)i * kHistThreads + threadIdx.x;
                if (p < count) atomicAdd(&s_hist[(from[p] >> shift) & (kRadix - 1)], 1);
            }
        }
    } else {
#pragma unroll 1
        for (int i0 = 0; i0 < kRounds; i0 += kBatch) {
            Raw raw[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; i++) raw[i] = load_raw<MODE>(s, base + (int64_t)(i0 + i) * kHistThreads + threadIdx.x, count);   // all loads in flight
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
                const Elem e = finish_elem<MODE>(s, base + (int64_t)(i0 + i) * kHistThreads + threadIdx.x, count, raw[i]);
                if (e.valid) atomicAdd(&s_hist[digit_of(e, shift, from_idx)], 1);
            }
        }
    }
    __syncthreads();
    matrix[(int64_t)blockIdx.x * kRadix + threadIdx.x] = s_hist[threadIdx.x];   // [tile][digit]: one coalesced row
}

// First-pass counts of BOTH formats from one read of the COO list (mode 1): by destination and by source.
template <int ITEMS>
__global__ void __launch_bounds__(kHistThreads) sort_hist_both_kernel(SortSrc s, int* __restrict__ by_dst, int* __restrict__ by_src) {
    __shared__ int s_hist[2][kRadix];
    constexpr int kSortTile = kSortThreads * ITEMS;
    constexpr int kRounds = ITEMS;
    constexpr int kBatch = 8;
    static_assert(kRounds % kBatch == 0, "a tile is read in whole batches");
    s_hist[0][threadIdx.x] = 0;
    s_hist[1][threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    const int64_t count = list_count(s);
    s.coo_w = nullptr;
    s.loop_w = nullptr;
#pragma unroll 1
    for (int i0 = 0; i0 < kRounds; i0 += kBatch) {
        Raw raw[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; i++) raw[i] = load_raw<1>(s, base + (int64_t)(i0 + i) * kHistThreads + threadIdx.x, count);
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
            const Elem e = finish_elem<1>(s, base + (int64_t)(i0 + i) * kHistThreads + threadIdx.x, count, raw[i]);
            if (e.valid) {
                const int src = s.by == 0 ? e.key : e.idx, dst = s.by == 0 ? e.idx : e.key;
                atomicAdd(&s_hist[0][dst & (kRadix - 1)], 1);
                atomicAdd(&s_hist[1][src & (kRadix - 1)], 1);
            }
        }
    }
    __syncthreads();
    by_dst[(int64_t)blockIdx.x * kRadix + threadIdx.x] = s_hist[0][threadIdx.x];
    by_src[(int64_t)blockIdx.x * kRadix + threadIdx.x] = s_hist[1][threadIdx.x];
}

struct SortDst {
    int32_t* key;   // may be null on the last pass when keys are not needed
    int32_t* idx;
    float* w;
};

// Stable scatter of one tile.  Element order inside the tile is (warp, round, lane), which is the
// order of the source list because warp w reads one contiguous range of 32 * kSortItems entries.
// HAS_W = false: every weight is 1 (no input weights), so the sort moves (key, index) pairs only and
// the caller writes the weights afterwards; a third less traffic per pass.
template <bool HAS_W, int MODE, int ITEMS>
__global__ void __launch_bounds__(kSortThreads, ITEMS == kItemsMany ? 3 : 4) sort_scatter_kernel(SortSrc s, SortDst d, int shift, int from_idx,
                                                                                                const int* __restrict__ matrix) {
    constexpr int kSortItems = ITEMS;
    constexpr int kSortTile = kSortThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char smem[];
    int2* s_pair = reinterpret_cast<int2*>(smem);                      // [kSortTile] (key, index): one 8-byte access per element
    int* s_whist = reinterpret_cast<int*>(s_pair + kSortTile);         // [kSortWarps][kRadix]
    int* s_gbase = s_whist + kSortWarps * kRadix;                      // [kRadix] global offset of a digit for this tile
    int* s_scan = s_gbase + kRadix;                                    // [32]
    float* s_w = reinterpret_cast<float*>(s_scan + 32);                // [kSortTile], HAS_W only
    __shared__ int s_total;

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t count = list_count(s);
    const int64_t wbase = (int64_t)blockIdx.x * kSortTile + (int64_t)wid * (32 * kSortItems);
    static_assert(kSortThreads == kRadix, "one thread per digit");
    const int tile_first = matrix[(int64_t)blockIdx.x * kRadix + threadIdx.x];   // this tile's global start of digit `threadIdx.x`: fetched first, needed last
    int32_t key[kSortItems], idx[kSortItems];
    float wt[HAS_W ? kSortItems : 1];
    unsigned valid = 0;
    // every load of the tile first (independent, all in flight), the ranking rounds after them
    if (MODE == 0) {
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const int64_t p = wbase + r * 32 + lane;
            const bool in = p < count;
            key[r] = in ? s.key[p] : 0;
            idx[r] = in ? s.idx[p] : 0;
            if (HAS_W) wt[r] = in ? s.w[p] : 0.f;
            valid |= in ? 1u << r : 0u;
        }
    } else {
        Raw raw[kSortItems];
#pragma unroll
        for (int r = 0; r < kSortItems; r++) raw[r] = load_raw<MODE>(s, wbase + r * 32 + lane, count);
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const Elem e = finish_elem<MODE>(s, wbase + r * 32 + lane, count, raw[r]);
            key[r] = e.key; idx[r] = e.idx;
            if (HAS_W) wt[r] = e.w;
            valid |= e.valid ? 1u << r : 0u;
        }
    }
    int* my_hist = s_whist + wid * kRadix;
#pragma unroll
    for (int i = 0; i < kRadix / 32; i++) my_hist[i * 32 + lane] = 0;
    __syncwarp();
    const unsigned lt_mask = (1u << lane) - 1u;
    // Ranking: lanes with the same digit find each other (by match mask or votes), the first of them takes the group's
    // places with ONE shared-memory atomic and hands the start round.  The rounds' atomics are issued one behind
    // the other and their results picked up afterwards, so a round does not wait for the one before it (a
    // read, a warp barrier, a write and another warp barrier per round were a chain of eight shared-memory
    // latencies: 2.05 -> 1.94 ms per pass of 285 M pairs; with the votes below 1.65).
    // place of an element: start of its group (valid in the group's first lane until it is handed round) in the low
    // 16 bits, that lane's number and the elements before this one in the bytes above - one register per element
    static_assert(kSortTile <= 1 << 16, "tile slots are kept in 16 bits");
    unsigned place[kSortItems];
    auto digit = [&](int r) { return ((unsigned)(from_idx ? idx[r] : key[r]) >> shift) & (kRadix - 1); };
    auto rank = [&](int r, unsigned dg, bool ok, unsigned peers) {
        place[r] = (unsigned)(__ffs(peers) - 1) << 16 | (unsigned)__popc(peers & lt_mask) << 24;
        if (ok && (peers & lt_mask) == 0) place[r] += (unsigned)atomicAdd(&my_hist[dg], __popc(peers));
        __syncwarp();
    };
    // Lanes with this lane's digit: a match mask, one step per distinct value among the lanes, or one vote per digit bit.
    // On shuffled edges (25 values in 32 lanes) the match kept its pipe 82 % busy and set the pace of the whole pass;
    // a list that is sorted already has a few runs in 32 lanes and is ranked faster by it (20 M edges sorted by
    // destination, three passes: 0.48 ms, 0.57 with votes).  The warp's first 32 elements decide for all its rounds.
    // With weights to carry it made no difference.
    bool runs = false;
    if (!HAS_W) {
        const unsigned left = __shfl_up_sync(kFull, digit(0), 1);
        runs = __popc(__ballot_sync(kFull, lane == 0 || digit(0) != left)) <= kMatchRuns;
    }
    if (runs) {
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const bool ok = (valid >> r) & 1u;
            const unsigned dg = digit(r);
            rank(r, dg, ok, __match_any_sync(kFull, ok ? dg : (unsigned)kRadix));
        }
    } else {
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const bool ok = (valid >> r) & 1u;
            const unsigned dg = digit(r);
            unsigned peers = __ballot_sync(kFull, ok);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const unsigned bit = (dg >> b) & 1u;
                peers &= __ballot_sync(kFull, bit) ^ (bit - 1u);
            }
            rank(r, dg, ok, peers);
        }
    }
#pragma unroll
    for (int r = 0; r < kSortItems; r++)
        place[r] = (__shfl_sync(kFull, place[r], (place[r] >> 16) & 31u) & 0xffffu) + (place[r] >> 24);
    __syncthreads();
    // one thread per digit: exclusive prefix over warps, tile total
    {
        // per warp and digit: first tile slot of that warp's elements of the digit (digit start + the earlier
        // warps' counts), so that staging needs one look-up per element
        const int dgt = threadIdx.x;
        int cnt_w[kSortWarps];
        int run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
            cnt_w[w] = s_whist[w * kRadix + dgt];
            run += cnt_w[w];
        }
        const int first = block_exclusive_scan(run, &s_total, s_scan);
        int at = first;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
            s_whist[w * kRadix + dgt] = at;
            at += cnt_w[w];
        }
        s_gbase[dgt] = tile_first - first;  // global position = gbase + tile slot
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        if ((valid >> r) & 1u) {
            const int q = my_hist[((from_idx ? idx[r] : key[r]) >> shift) & (kRadix - 1)] + (int)place[r];
            s_pair[q] = make_int2(key[r], idx[r]);
            if (HAS_W) s_w[q] = wt[r];
        }
    }
    __syncthreads();
    const int total = s_total;
#pragma unroll 4
    for (int q = threadIdx.x; q < total; q += kSortThreads) {
        const int2 e = s_pair[q];
        const int64_t g = (int64_t)s_gbase[((from_idx ? e.y : e.x) >> shift) & (kRadix - 1)] + q;   // the digit again, from the element
        if (d.key) d.key[g] = e.x;
        d.idx[g] = e.y;
        if (HAS_W) d.w[g] = s_w[q];
    }
}

constexpr size_t scatter_smem(bool has_w, int items) {
    return (size_t)kSortThreads * items * (has_w ? 12 : 8) + sizeof(int) * (kSortWarps * kRadix + kRadix + 32);
}

typedef void (*ScatterFn)(SortSrc, SortDst, int, int, const int*);
typedef void (*HistFn)(SortSrc, int, int, int*);
// The instantiations: a list with weights takes kItemsFew, a mirrored list (mode 2) always has weights.
static ScatterFn scatter_fn(bool has_w, int mode, int items) {
    if (has_w)
        return mode == 0 ? sort_scatter_kernel<true, 0, kItemsFew> : mode == 1 ? sort_scatter_kernel<true, 1, kItemsFew>
                                                                               : sort_scatter_kernel<true, 2, kItemsFew>;
    if (mode == 2) return nullptr;
    if (items == kItemsFew) return mode == 0 ? sort_scatter_kernel<false, 0, kItemsFew> : sort_scatter_kernel<false, 1, kItemsFew>;
    return mode == 0 ? sort_scatter_kernel<false, 0, kItemsMany> : sort_scatter_kernel<false, 1, kItemsMany>;
}
static HistFn hist_fn(int mode, int items) {
    if (mode == 2) return sort_hist_kernel<2, kItemsFew>;
    if (items == kItemsFew) return mode == 0 ? sort_hist_kernel<0, kItemsFew> : sort_hist_kernel<1, kItemsFew>;
    return mode == 0 ? sort_hist_kernel<0, kItemsMany> : sort_hist_kernel<1, kItemsMany>;
}

// ------------------------------------------------------------------------------- small kernels
// off[k] = first position whose key is >= k, for k in [0, n]; keys sorted, E entries.
// Each thread takes four groups of four consecutive positions, a block's width apart, and issues all their loads
// before it looks at one (285 M keys: 0.39 -> 0.38 ms; the runs of empty rows, written one by one, are the rest).
// GAPS: rows may be empty, in long runs even (users below, items above: written by one thread, 4 M empty rows took
// 15 ms).  Then a thread ends its run at the next multiple of kGapTile rows, and one warp per tile, in the first
// `fill_blocks` blocks, looks up its first row's offset and writes the run that row is in up to the tile's end.
constexpr int kOffThreads = 256;
constexpr int kOffGroups = 4;
constexpr int64_t kOffTile = (int64_t)kOffThreads * kOffGroups * 4;
constexpr int kGapTile = 512;      // a power of two

__device__ void fill_tile_start(const int32_t* __restrict__ key, int64_t E, int64_t n, int64_t v0, int32_t* __restrict__ off) {
    const int lane = lane_id();
    // first position with a key >= v0: 32 probes at once cut the range by 33
    int64_t lo = 0, hi = E;
    while (lo < hi) {
        const int64_t len = hi - lo;
        const unsigned below = __ballot_sync(kFull, __ldg(key + lo + (lane + 1) * len / 33) < v0);
        const int c = __popc(below);        // keys are sorted: the first c probes
        hi = c < 32 ? lo + (c + 1) * len / 33 : hi;
        lo = c > 0 ? lo + c * len / 33 + 1 : lo;
    }
    int64_t last = lo < E ? (int64_t)__ldg(key + lo) : n;
    if (last > v0 + kGapTile - 1) last = v0 + kGapTile - 1;
    for (int64_t v = v0 + lane; v <= last; v += 32) off[v] = (int32_t)lo;
}

template <bool GAPS>
__global__ void __launch_bounds__(kOffThreads) offsets_from_sorted_keys(const int32_t* __restrict__ key, int64_t E_host,
                                                                        const unsigned long long* __restrict__ dcount, int64_t n,
                                                                        int32_t* __restrict__ off, unsigned fill_blocks) {
    const int64_t E = dcount ? (int64_t)*dcount : E_host;
    if (GAPS && blockIdx.x < fill_blocks) {
        const int64_t v0 = ((int64_t)blockIdx.x * (kOffThreads / 32) + threadIdx.x / 32) * kGapTile;
        if (v0 <= n) fill_tile_start(key, E, n, v0, off);
        return;
    }
    const int64_t base = (int64_t)(GAPS ? blockIdx.x - fill_blocks : blockIdx.x) * kOffTile + 4 * threadIdx.x;
    const bool vec = reinterpret_cast<uintptr_t>(key) % 16 == 0;
    int4 k4[kOffGroups];
    int32_t before[kOffGroups];
#pragma unroll
    for (int g = 0; g < kOffGroups; g++) {
        const int64_t j = base + (int64_t)g * kOffThreads * 4;
        before[g] = j > 0 && j <= E ? __ldg(key + j - 1) : -1;
        k4[g] = make_int4(0, 0, 0, 0);
        if (vec && j + 4 <= E) {
            k4[g] = __ldg(reinterpret_cast<const int4*>(key + j));
        } else {
            if (j < E) k4[g].x = __ldg(key + j);
            if (j + 1 < E) k4[g].y = __ldg(key + j + 1);
            if (j + 2 < E) k4[g].z = __ldg(key + j + 2);
            if (j + 3 < E) k4[g].w = __ldg(key + j + 3);
        }
    }
#pragma unroll
    for (int g = 0; g < kOffGroups; g++) {
        const int64_t j0 = base + (int64_t)g * kOffThreads * 4;
        int64_t prev = before[g];
        const int32_t k[4] = {k4[g].x, k4[g].y, k4[g].z, k4[g].w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t j = j0 + i;
            if (j > E) break;
            const int64_t hi = j == E ? n : k[i];
            const int64_t border = prev | (kGapTile - 1);      // the last row before the next tile
            const int64_t end = GAPS && border < hi ? border : hi;
            for (int64_t v = prev + 1; v <= end; v++) off[v] = (int32_t)j;
            prev = hi;
        }
    }
}
// count: the entries, or their upper bound where dcount holds the number.  `gaps`: rows may be empty (with a loop on
// every node none is).  A run of two tiles is written by one thread sooner than a search ends.
static int launch_offsets(const int32_t* key, int64_t count, const unsigned long long* dcount, int64_t n, int32_t* off, bool gaps,
                          cudaStream_t st) {
    const unsigned blocks = (unsigned)(count / kOffTile + 1);              // positions 0 .. count
    if (gaps && n >= 2 * kGapTile) {
        const int64_t tiles = n / kGapTile + 1;                            // rows 0 .. n
        const unsigned fill = (unsigned)((tiles + kOffThreads / 32 - 1) / (kOffThreads / 32));
        offsets_from_sorted_keys<true><<<fill + blocks, kOffThreads, 0, st>>>(key, count, dcount, n, off, fill);
    } else {
        offsets_from_sorted_keys<false><<<blocks, kOffThreads, 0, st>>>(key, count, dcount, n, off, 0);
    }
    JG_LAUNCH_CHECK();
    return JG_OK;
}

__global__ void set_count_kernel(unsigned long long* p, unsigned long long v) { *p = v; }

static int launch_set_count(unsigned long long* p, unsigned long long v, cudaStream_t st) {
    set_count_kernel<<<1, 1, 0, st>>>(p, v);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

// Weight of the loop appended for node v: the fill value, or the weight of the LAST (v,v) input
// entry (an indexed assignment keeps the last write, utils/loop.py:131-133).
__global__ void last_loop_index_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t e0,
                                       int* __restrict__ last) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < e0; i += (int64_t)gridDim.x * blockDim.x)
        if (src[i] == dst[i]) atomicMax(&last[src[i]], (int)i);
}
__global__ void loop_weight_kernel(const int* __restrict__ last, const float* __restrict__ w, float fill, int64_t n,
                                   float* __restrict__ loop_w) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) loop_w[v] = last[v] >= 0 ? (w ? w[last[v]] : 1.f) : fill;
}

// deg[v] = sum of the raw weights of column v; dis = deg^-1/2 correctly rounded through double.  Columns of up to
// kLongColumn entries are added sequentially in list order, the order a host scatter-add takes: by one thread up to
// kThreadColumn entries, else by a warp that reads 32 entries at a time and adds them one by one.  A longer column
// is added by a block - every thread a strided part, then a fixed tree - which is closer to the exact sum than the
// sequential order.  With one thread per column whatever its length, a 30 M-edge weighted R-MAT list spent 1.86 of
// the conversion's 4.5 ms here, behind the threads that own the hubs.
// Columns beyond one thread's share are listed: warp columns from the front of `list`, block columns from its back,
// count[0] and count[1] of them (zeroed by the launcher), so that neighbouring hubs spread over the device.
constexpr int kThreadColumn = 64;
constexpr int kLongColumn = 4096;
constexpr int kDegThreads = 256;
__device__ __forceinline__ float inv_sqrt_degree(float deg) { return (float)(1.0 / sqrt((double)deg)); }

__global__ void __launch_bounds__(kDegThreads) degree_kernel(const int32_t* __restrict__ off, const float* __restrict__ w, int64_t n,
                                                             int unit, float* __restrict__ dis, int* __restrict__ list,
                                                             int* __restrict__ count) {
    const int64_t v = (int64_t)blockIdx.x * kDegThreads + threadIdx.x;
    if (v >= n) return;
    const int32_t s = off[v], e = off[v + 1];
    float deg = 0.f;
    if (unit) {
        deg = (float)(e - s);  // exact while the count stays below 2^24, as sequential adds of 1.0f are
        if (e - s > (1 << 24)) {
            deg = 0.f;
            for (int32_t j = s; j < e; j++) deg = __fadd_rn(deg, 1.f);
        }
    } else if (e - s <= kThreadColumn) {
        for (int32_t j = s; j < e; j++) deg = __fadd_rn(deg, __ldg(w + j));
    } else {
        if (e - s <= kLongColumn) list[atomicAdd(&count[0], 1)] = (int)v;
        else list[n - 1 - atomicAdd(&count[1], 1)] = (int)v;
        return;
    }
    dis[v] = inv_sqrt_degree(deg);
}

__global__ void __launch_bounds__(kDegThreads) degree_listed_kernel(const int32_t* __restrict__ off, const float* __restrict__ w,
                                                                    int64_t n, float* __restrict__ dis, const int* __restrict__ list,
                                                                    const int* __restrict__ count) {
    __shared__ float s_part[kDegThreads / 32];
    const int lane = threadIdx.x & 31;
    const int n_warp = count[0], n_block = count[1];
    for (int i = blockIdx.x; i < n_block; i += gridDim.x) {
        const int64_t v = list[n - 1 - i];
        const int64_t s = off[v], e = off[v + 1];
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] = 0.f;
        for (int64_t j = s + threadIdx.x; j < e; j += 8 * kDegThreads) {
            float t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = j + k * kDegThreads < e ? __ldg(w + j + k * kDegThreads) : 0.f;
#pragma unroll
            for (int k = 0; k < 8; k++) acc[k] += t[k];
        }
        float sum = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
        if (lane == 0) s_part[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            float deg = 0.f;
#pragma unroll
            for (int q = 0; q < kDegThreads / 32; q++) deg += s_part[q];
            dis[v] = inv_sqrt_degree(deg);
        }
        __syncthreads();
    }
    const int warps = (int)gridDim.x * (kDegThreads / 32);
    for (int i = (int)blockIdx.x * (kDegThreads / 32) + (threadIdx.x >> 5); i < n_warp; i += warps) {
        const int v = list[i];
        const int64_t s = off[v], e = off[v + 1];
        float deg = 0.f;
        float next = s + lane < e ? __ldg(w + s + lane) : 0.f;
        for (int64_t j = s; j < e; j += 32) {
            const float t = next;
            next = j + 32 + lane < e ? __ldg(w + j + 32 + lane) : 0.f;
#pragma unroll
            for (int k = 0; k < 32; k++) deg = __fadd_rn(deg, __shfl_sync(kFull, t, k));   // + 0 beyond the column's end
        }
        if (lane == 0) dis[v] = inv_sqrt_degree(deg);
    }
}

// w'[j] = (dis[source] * w[j]) * dis[destination]  (nn/conv/gcn_conv.py:37); key is the segment
// owner, idx the other endpoint; key_is_dst tells which is which.
__global__ void norm_weight_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ idx, float* __restrict__ w,
                                   const float* __restrict__ dis, const unsigned long long* __restrict__ dcount,
                                   int key_is_dst, int unit) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= (int64_t)*dcount) return;
    const int32_t k = key[j], o = idx[j];
    const float ds = dis[key_is_dst ? o : k], dd = dis[key_is_dst ? k : o];
    w[j] = __fmul_rn(__fmul_rn(ds, unit ? 1.f : w[j]), dd);   // unit: the sort did not carry the (all-one) weights
}

// Four entries per thread (16-byte loads and store; all three arrays 16-byte aligned): with one entry per
// thread the pass was bound by occupancy times a chain of three dependent latencies (count, endpoints, dis).
__global__ void __launch_bounds__(256) norm_weight_vec_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ idx,
                                                              float* __restrict__ w, const float* __restrict__ dis,
                                                              const unsigned long long* __restrict__ dcount, int key_is_dst, int unit) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t count = (int64_t)*dcount;
    const int64_t j = 4 * t;
    if (j >= count) return;
    if (j + 4 <= count) {
        const int4 k = reinterpret_cast<const int4*>(key)[t], o = reinterpret_cast<const int4*>(idx)[t];
        float4 v = unit ? make_float4(1.f, 1.f, 1.f, 1.f) : reinterpret_cast<const float4*>(w)[t];
        const int4 a = key_is_dst ? o : k, b = key_is_dst ? k : o;     // a: sources, b: destinations
        const float s0 = dis[a.x], s1 = dis[a.y], s2 = dis[a.z], s3 = dis[a.w];
        const float d0 = dis[b.x], d1 = dis[b.y], d2 = dis[b.z], d3 = dis[b.w];
        v.x = __fmul_rn(__fmul_rn(s0, v.x), d0); v.y = __fmul_rn(__fmul_rn(s1, v.y), d1);
        v.z = __fmul_rn(__fmul_rn(s2, v.z), d2); v.w = __fmul_rn(__fmul_rn(s3, v.w), d3);
        reinterpret_cast<float4*>(w)[t] = v;
    } else {
        for (int64_t i = j; i < count; i++) {
            const int32_t kk = key[i], oo = idx[i];
            const float ds = dis[key_is_dst ? oo : kk], dd = dis[key_is_dst ? kk : oo];
            w[i] = __fmul_rn(__fmul_rn(ds, unit ? 1.f : w[i]), dd);
        }
    }
}

static int launch_norm_weights(const int32_t* key, const int32_t* idx, float* w, const float* dis, const unsigned long long* dcount,
                               int key_is_dst, int unit, int64_t cap, cudaStream_t st) {
    if (cap <= 0) return JG_OK;
    if ((reinterpret_cast<uintptr_t>(key) | reinterpret_cast<uintptr_t>(idx) | reinterpret_cast<uintptr_t>(w)) % 16 == 0)
        norm_weight_vec_kernel<<<(unsigned)(((cap + 3) / 4 + 255) / 256), 256, 0, st>>>(key, idx, w, dis, dcount, key_is_dst, unit);
    else
        norm_weight_kernel<<<(unsigned)((cap + 255) / 256), 256, 0, st>>>(key, idx, w, dis, dcount, key_is_dst, unit);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

// keep[i] = 1 for input entries that are not (v,v)
__global__ void keep_flags_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t e0,
                                  int* __restrict__ keep) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < e0) keep[i] = src[i] != dst[i];
}

// Normalised COO list in the reference's order: kept entries in input order, then one loop per node.
__global__ void write_norm_coo_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                      const float* __restrict__ w, const float* __restrict__ loop_w,
                                      const int* __restrict__ pos, const float* __restrict__ dis, int64_t e0, int64_t n,
                                      const unsigned long long* __restrict__ total, int32_t* __restrict__ out_src,
                                      int32_t* __restrict__ out_dst, float* __restrict__ out_w) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t kept = (int64_t)*total - n;
    if (i < e0) {
        const int32_t a = src[i], b = dst[i];
        if (a != b) {
            const int64_t p = pos[i];
            out_src[p] = a;
            out_dst[p] = b;
            out_w[p] = __fmul_rn(__fmul_rn(dis[a], w ? w[i] : 1.f), dis[b]);
        }
    } else if (i < e0 + n) {
        const int32_t v = (int32_t)(i - e0);
        out_src[kept + v] = v;
        out_dst[kept + v] = v;
        out_w[kept + v] = __fmul_rn(__fmul_rn(dis[v], loop_w ? loop_w[v] : 1.f), dis[v]);
    }
}

// add_self_loops = false: entry i keeps its place, w' = (dis[src] * w) * dis[dst]
__global__ void norm_coo_plain_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                      const float* __restrict__ w, const float* __restrict__ dis, int64_t e0,
                                      int32_t* __restrict__ out_src, int32_t* __restrict__ out_dst, float* __restrict__ out_w) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= e0) return;
    const int32_t a = src[i], b = dst[i];
    out_src[i] = a;
    out_dst[i] = b;
    out_w[i] = __fmul_rn(__fmul_rn(dis[a], w ? w[i] : 1.f), dis[b]);
}

// ---- symmetrise + dedupe: first entry of every run of equal (row, col) pairs survives
__global__ void first_of_run_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ idx, int64_t m,
                                    int* __restrict__ flag) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < m) flag[j] = (j == 0) || key[j] != key[j - 1] || idx[j] != idx[j - 1];
    if (j == m) flag[j] = 0;
}
__global__ void compact_runs_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ idx,
                                    const float* __restrict__ w, const int* __restrict__ pos, int64_t m,
                                    int32_t* __restrict__ out_src, int32_t* __restrict__ out_dst,
                                    float* __restrict__ out_w, int64_t* __restrict__ out_count) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < m) {
        const bool first = (j == 0) || key[j] != key[j - 1] || idx[j] != idx[j - 1];
        if (first) {
            const int p = pos[j];
            out_src[p] = key[j];
            out_dst[p] = idx[j];
            out_w[p] = w[j];
        }
    }
    if (j == m) *out_count = pos[m];
}

// ---- 1-D row partition: split a shard's in-edges into interior (source owned) and halo (remote)
__global__ void interior_flags_kernel(const int32_t* __restrict__ idx, int64_t nnz, int32_t lo, int32_t hi,
                                      int* __restrict__ flag) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nnz) flag[e] = idx[e] >= lo && idx[e] < hi;
    if (e == nnz) flag[e] = 0;
}

// pos[e] = number of interior entries before e (exclusive scan of the flags, nnz + 1 entries).
__global__ void split_write_kernel(const int32_t* __restrict__ idx, const float* __restrict__ w,
                                   const int* __restrict__ pos, int64_t nnz, int32_t lo, int32_t hi,
                                   int32_t* __restrict__ int_idx, float* __restrict__ int_w,
                                   int32_t* __restrict__ halo_idx, float* __restrict__ halo_w) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const int32_t s = idx[e];
    const int p = pos[e];
    if (s >= lo && s < hi) {
        int_idx[p] = s - lo;     // interior sources are addressed inside the shard's own rows
        int_w[p] = w[e];
    } else {
        halo_idx[e - p] = s;     // halo sources keep their global id
        halo_w[e - p] = w[e];
    }
}

__global__ void split_offsets_kernel(const int32_t* __restrict__ off, const int* __restrict__ pos, int64_t n_rows,
                                     int32_t* __restrict__ int_off, int32_t* __restrict__ halo_off,
                                     int64_t* __restrict__ counts) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v > n_rows) return;
    const int32_t o = off[v];
    const int p = pos[o];
    int_off[v] = p;
    halo_off[v] = o - p;
    if (v == n_rows) {
        counts[0] = p;
        counts[1] = o - p;
    }
}

__global__ void iota_kernel(int* p, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = (int)i;
}

__global__ void fill_int_kernel(int* p, int v, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// ------------------------------------------------------------------------------- host driver
static int bits_for(int64_t n) {
    int b = 1;
    while (b < 31 && ((int64_t)1 << b) < n) b++;
    return b;
}

struct ConvertWs {
    int32_t *key[2], *idx[2];
    float* w[2];
    int* matrix;
    int* matrix2;     // first-pass counts of the second format, taken with the first's
    int* scan_sums;
    float* dis;
    float* loop_w;
    int* last_loop;
    int* deg_count;      // [2] columns listed by degree_kernel
    unsigned long long* kept;
    size_t bytes;
};

static ConvertWs carve_convert(void* ws, int64_t cap, int64_t n) {
    Carver c(ws);
    ConvertWs v;
    for (int b = 0; b < 2; b++) {
        v.key[b] = c.take<int32_t>(cap);
        v.idx[b] = c.take<int32_t>(cap);
        v.w[b] = c.take<float>(cap);
    }
    const int64_t tiles = sort_tiles(cap, kItemsFew) + 1;   // the form with the most tiles
    v.matrix = c.take<int>((size_t)tiles * kRadix);
    v.matrix2 = c.take<int>((size_t)tiles * kRadix);
    v.scan_sums = c.take<int>((size_t)((tiles + kChunkTiles - 1) / kChunkTiles + 1) * kRadix);
    v.dis = c.take<float>(n + 1);
    v.loop_w = c.take<float>(n + 1);
    v.last_loop = c.take<int>(n + 1);
    v.deg_count = c.take<int>(2);
    v.kept = c.take<unsigned long long>(1);
    v.bytes = c.total();
    return v;
}

// Sorts the (virtual) list described by `first` into (keys, out_idx, out_w), stable on the key;
// canonical additionally orders the entries of one key by their index.  `kept` (device) is the
// element count after a first pass that drops entries, or null when first.count is exact.
// *sorted_key receives the buffer holding the sorted keys.
// carry_w = false (all weights are 1): out_w is left untouched, the caller fills it.
// counted: the first pass's per-tile digit counts when the caller has them already (else null);
// total (device, or null) receives the number of entries the first pass keeps.
static int radix_sort(SortSrc first, int64_t n, int canonical, const unsigned long long* kept, ConvertWs& ws,
                      int32_t* out_idx, float* out_w, int32_t** sorted_key, cudaStream_t st, bool carry_w = true,
                      int* counted = nullptr, unsigned long long* total = nullptr) {
    static bool attr_set[64] = {false};
    int dev = 0;
    JG_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        for (int v = 0; v < 12; v++) {
            const bool has_w = v >= 6;
            const int mode = v % 3, items = v % 6 >= 3 ? kItemsMany : kItemsFew;
            ScatterFn fn = has_w && items == kItemsMany ? nullptr : scatter_fn(has_w, mode, items);
            if (fn)
                JG_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)scatter_smem(has_w, items)));
        }
        attr_set[dev] = true;
    }
    const int bits = bits_for(n);
    const int key_passes = (bits + 7) / 8;
    const int total_passes = canonical ? 2 * key_passes : key_passes;
    JG_CHECK_ARG(first.mode != 2 || carry_w, JG_EINVAL, "radix_sort: a mirrored list carries weights");
    const int items = sort_items(first.count, carry_w);
    const int64_t tiles = sort_tiles(first.count, items);  // upper bound for every pass
    SortSrc src = first;
    int cur = 0;
    *sorted_key = ws.key[0];
    if (tiles == 0) return JG_OK;
    for (int p = 0; p < total_passes; p++) {
        const int from_idx = canonical && p < key_passes;
        const int shift = 8 * (canonical && !from_idx ? p - key_passes : p);
        int* matrix = ws.matrix;
        if (p == 0 && counted) {
            matrix = counted;
        } else {
            hist_fn(src.mode, items)<<<(unsigned)tiles, kHistThreads, 0, st>>>(src, shift, from_idx, matrix);
            JG_LAUNCH_CHECK();
        }
        if (tiles <= kChunkTiles) {
            colscan_small<<<1, kRadix, 0, st>>>(matrix, (int)tiles, p == 0 ? total : nullptr);
            JG_LAUNCH_CHECK();
        } else {
            const int64_t chunks = (tiles + kChunkTiles - 1) / kChunkTiles;
            colscan_chunk_sums<<<(unsigned)chunks, kRadix, 0, st>>>(matrix, tiles, ws.scan_sums);
            JG_LAUNCH_CHECK();
            colscan_chunks<<<1, kRadix, 0, st>>>(ws.scan_sums, chunks, p == 0 ? total : nullptr);
            JG_LAUNCH_CHECK();
            colscan_apply<<<(unsigned)chunks, kRadix, 0, st>>>(matrix, tiles, ws.scan_sums);
            JG_LAUNCH_CHECK();
        }
        const bool last = p == total_passes - 1;
        SortDst dst;
        dst.key = ws.key[cur];
        dst.idx = last ? out_idx : ws.idx[cur];
        dst.w = carry_w ? (last ? out_w : ws.w[cur]) : nullptr;
        scatter_fn(carry_w, src.mode, items)<<<(unsigned)tiles, kSortThreads, scatter_smem(carry_w, items), st>>>(src, dst, shift, from_idx, matrix);
        JG_LAUNCH_CHECK();
        *sorted_key = dst.key;
        SortSrc nxt = {};
        nxt.mode = 0;
        nxt.key = dst.key; nxt.idx = dst.idx; nxt.w = dst.w;
        nxt.count = first.count;
        nxt.dcount = kept;
        src = nxt;
        cur ^= 1;
    }
    return JG_OK;
}

static inline unsigned blocks_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace jg

using namespace jg;

extern "C" {

size_t jg_convert_workspace_bytes(int64_t n_edges, int64_t n_nodes) {
    if (n_edges < 0 || n_nodes < 0) return 0;
    return carve_convert(nullptr, n_edges + n_nodes, n_nodes).bytes;
}

int jg_coo_to_compressed(const int32_t* edge_index, const float* w, int64_t n_edges, int64_t n_nodes, int by,
                         int canonical, int32_t* out_idx, int32_t* out_off, float* out_w, void* workspace,
                         size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(n_edges >= 0 && n_nodes >= 0, JG_EINVAL, "coo_to_compressed: negative size");
    JG_CHECK_ARG(by == 0 || by == 1, JG_EINVAL, "coo_to_compressed: by must be 0 (source) or 1 (destination)");
    JG_CHECK_ARG(out_off, JG_EINVAL, "coo_to_compressed: null offsets");
    JG_CHECK_ARG(n_edges == 0 || (edge_index && out_idx && out_w), JG_EINVAL, "coo_to_compressed: null array");
    JG_CHECK_ARG(n_edges <= INT32_MAX - 1 && n_nodes < INT32_MAX, JG_ESHAPE, "coo_to_compressed: sizes beyond int32");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_convert_workspace_bytes(n_edges, n_nodes), JG_EWORKSPACE,
                 "coo_to_compressed: workspace %zu < %zu", workspace_bytes, jg_convert_workspace_bytes(n_edges, n_nodes));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ConvertWs ws = carve_convert(workspace, n_edges + n_nodes, n_nodes);
    SortSrc first = {};
    first.mode = 1;
    first.coo_src = edge_index;
    first.coo_dst = edge_index + n_edges;
    first.coo_w = w;
    first.e0 = n_edges;
    first.by = by;
    first.count = n_edges;
    int32_t* skey = nullptr;
    const bool carry_w = w != nullptr;
    int rc = radix_sort(first, n_nodes, canonical, nullptr, ws, out_idx, out_w, &skey, st, carry_w);
    if (rc != JG_OK) return rc;
    if (!carry_w && n_edges > 0) {   // no input weights: every output weight is 1.0f
        fill_int_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(reinterpret_cast<int*>(out_w), 0x3f800000, n_edges);
        JG_LAUNCH_CHECK();
    }
    return launch_offsets(skey, n_edges, nullptr, n_nodes, out_off, true, st);
}

int jg_group_edges(const int32_t* node, int64_t n_edges, int64_t n_nodes, int32_t* out_edge, int32_t* out_off, float* out_ones,
                   void* workspace, size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(n_edges >= 0 && n_nodes >= 0, JG_EINVAL, "group_edges: negative size");
    JG_CHECK_ARG(out_off && (n_edges == 0 || (node && out_edge)), JG_EINVAL, "group_edges: null array");
    JG_CHECK_ARG(n_edges <= INT32_MAX - 1 && n_nodes < INT32_MAX, JG_ESHAPE, "group_edges: sizes beyond int32");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_convert_workspace_bytes(n_edges, n_nodes), JG_EWORKSPACE,
                 "group_edges: workspace %zu < %zu", workspace_bytes, jg_convert_workspace_bytes(n_edges, n_nodes));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ConvertWs ws = carve_convert(workspace, n_edges + n_nodes, n_nodes);
    SortSrc first = {};
    // the second buffer's indices are written only after the first pass has read the positions from there
    first.mode = 1;
    first.coo_src = node;
    first.coo_dst = ws.idx[1];
    if (n_edges > 0) {
        iota_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(ws.idx[1], n_edges);
        JG_LAUNCH_CHECK();
    }
    first.e0 = n_edges;
    first.by = 0;
    first.count = n_edges;
    int32_t* skey = nullptr;
    int rc = radix_sort(first, n_nodes, 0, nullptr, ws, out_edge, nullptr, &skey, st, false);
    if (rc != JG_OK) return rc;
    if (out_ones && n_edges > 0) {
        fill_int_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(reinterpret_cast<int*>(out_ones), 0x3f800000, n_edges);
        JG_LAUNCH_CHECK();
    }
    return launch_offsets(skey, n_edges, nullptr, n_nodes, out_off, true, st);
}

int jg_gcn_norm_compressed(const int32_t* edge_index, const float* w, int64_t n_edges, int64_t n_nodes, float fill,
                           int add_self_loops, int canonical, int32_t* csc_idx, int32_t* csc_off, float* csc_w,
                           int32_t* csr_idx, int32_t* csr_off, float* csr_w, int64_t* out_count, void* workspace,
                           size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(n_edges >= 0 && n_nodes >= 0, JG_EINVAL, "gcn_norm_compressed: negative size");
    JG_CHECK_ARG(csc_idx && csc_off && csc_w && out_count, JG_EINVAL, "gcn_norm_compressed: CSC outputs and count are required");
    JG_CHECK_ARG((csr_idx && csr_off && csr_w) || (!csr_idx && !csr_off && !csr_w), JG_EINVAL,
                 "gcn_norm_compressed: CSR outputs must be all given or all null");
    JG_CHECK_ARG(n_edges == 0 || edge_index, JG_EINVAL, "gcn_norm_compressed: null edge_index");
    JG_CHECK_ARG(n_edges + n_nodes <= INT32_MAX - 1, JG_ESHAPE, "gcn_norm_compressed: sizes beyond int32");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_convert_workspace_bytes(n_edges, n_nodes), JG_EWORKSPACE,
                 "gcn_norm_compressed: workspace %zu < %zu", workspace_bytes, jg_convert_workspace_bytes(n_edges, n_nodes));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t cap = n_edges + n_nodes;
    ConvertWs ws = carve_convert(workspace, cap, n_nodes);
    const int32_t* src = edge_index;
    const int32_t* dst = edge_index + n_edges;
    const int grid = sm_count() * 8;

    const bool unit = (w == nullptr) && (fill == 1.0f || !add_self_loops);
    const float* loop_w = nullptr;
    if (!unit && n_nodes > 0 && add_self_loops) {
        fill_int_kernel<<<blocks_for(n_nodes, 256), 256, 0, st>>>(ws.last_loop, -1, n_nodes);
        JG_LAUNCH_CHECK();
        if (n_edges > 0) {
            last_loop_index_kernel<<<grid, 256, 0, st>>>(src, dst, n_edges, ws.last_loop);
            JG_LAUNCH_CHECK();
        }
        loop_weight_kernel<<<blocks_for(n_nodes, 256), 256, 0, st>>>(ws.last_loop, w, fill, n_nodes, ws.loop_w);
        JG_LAUNCH_CHECK();
        loop_w = ws.loop_w;
    }
    SortSrc first = {};
    first.mode = 1;
    first.coo_src = src; first.coo_dst = dst; first.coo_w = w; first.loop_w = loop_w;
    first.e0 = n_edges;
    first.n_loops = add_self_loops ? n_nodes : 0;
    first.drop_loops = add_self_loops ? 1 : 0;
    first.count = add_self_loops ? cap : n_edges;

    // destination-major (CSC), raw weights; degrees and dis from its segments
    int32_t* skey = nullptr;
    first.by = 1;
    int* counted = nullptr;
    if (csr_idx && !canonical && first.count > 0) {
        const int items = sort_items(first.count, !unit);
        auto kern = items == kItemsFew ? sort_hist_both_kernel<kItemsFew> : sort_hist_both_kernel<kItemsMany>;
        kern<<<(unsigned)sort_tiles(first.count, items), kHistThreads, 0, st>>>(first, ws.matrix, ws.matrix2);
        JG_LAUNCH_CHECK();
        counted = ws.matrix;
    }
    // ws.kept, the entries that survive (non-loop input entries + one loop per node; without self-loops the list as
    // given), is the total of the first pass's counts
    int rc = first.count > 0 ? JG_OK : launch_set_count(ws.kept, 0, st);
    if (rc != JG_OK) return rc;
    rc = radix_sort(first, n_nodes, canonical, ws.kept, ws, csc_idx, csc_w, &skey, st, !unit, counted, ws.kept);
    if (rc != JG_OK) return rc;
    rc = launch_offsets(skey, cap, ws.kept, n_nodes, csc_off, !add_self_loops, st);
    if (rc != JG_OK) return rc;
    if (n_nodes > 0) {
        int* list = ws.last_loop;      // free again: the loop weights have been taken
        if (!unit) JG_CUDA(cudaMemsetAsync(ws.deg_count, 0, 2 * sizeof(int), st));
        degree_kernel<<<blocks_for(n_nodes, kDegThreads), kDegThreads, 0, st>>>(csc_off, csc_w, n_nodes, unit ? 1 : 0, ws.dis, list, ws.deg_count);
        JG_LAUNCH_CHECK();
        if (!unit) {
            degree_listed_kernel<<<sm_count() * 4, kDegThreads, 0, st>>>(csc_off, csc_w, n_nodes, ws.dis, list, ws.deg_count);
            JG_LAUNCH_CHECK();
        }
    }
    rc = launch_norm_weights(skey, csc_idx, csc_w, ws.dis, ws.kept, 1, unit ? 1 : 0, cap, st);
    if (rc != JG_OK) return rc;
    if (csr_idx) {
        bool weights_done = false;
        if (canonical) {
            // The canonical CSC list is ordered by (destination, source); ONE stable sort of it by source gives
            // (source, destination), the canonical CSR, in half the passes of sorting the input again by both
            // keys.  The normalised weight of an entry is the same number in both formats, so it travels with
            // the entry (unit weights are not carried at all and are written afterwards, as for the CSC).
            SortSrc from_csc = {};
            from_csc.mode = 0;
            from_csc.key = csc_idx;                 // source of every entry, the new key
            from_csc.idx = skey;                    // its destination (the sorted keys of the CSC sort)
            from_csc.w = unit ? nullptr : csc_w;
            from_csc.count = first.count;
            from_csc.dcount = ws.kept;
            rc = radix_sort(from_csc, n_nodes, 0, ws.kept, ws, csr_idx, csr_w, &skey, st, !unit);
            weights_done = !unit;
        } else {
            first.by = 0;
            rc = radix_sort(first, n_nodes, canonical, ws.kept, ws, csr_idx, csr_w, &skey, st, !unit, counted ? ws.matrix2 : nullptr);
        }
        if (rc != JG_OK) return rc;
        rc = launch_offsets(skey, cap, ws.kept, n_nodes, csr_off, !add_self_loops, st);
        if (rc != JG_OK) return rc;
        if (!weights_done) {
            rc = launch_norm_weights(skey, csr_idx, csr_w, ws.dis, ws.kept, 0, unit ? 1 : 0, cap, st);
            if (rc != JG_OK) return rc;
        }
    }
    JG_CUDA(cudaMemcpyAsync(out_count, ws.kept, sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st));
    return JG_OK;
}


struct NormCooWs {
    void* convert;
    size_t convert_bytes;
    int32_t* tmp_idx;
    int32_t* tmp_off;
    float* tmp_w;
    int* pos;
    int* pos_sums;
    int64_t* count;
    size_t bytes;
};

static NormCooWs carve_norm_coo(void* ws, int64_t n_edges, int64_t n_nodes) {
    Carver c(ws);
    NormCooWs v;
    v.convert_bytes = jg_convert_workspace_bytes(n_edges, n_nodes);
    v.convert = c.take<unsigned char>(v.convert_bytes);
    v.tmp_idx = c.take<int32_t>(n_edges + n_nodes);
    v.tmp_off = c.take<int32_t>(n_nodes + 1);
    v.tmp_w = c.take<float>(n_edges + n_nodes);
    v.pos = c.take<int>(n_edges + 1);
    v.pos_sums = c.take<int>(scan_temp_ints(n_edges + 1));
    v.count = c.take<int64_t>(1);
    v.bytes = c.total();
    return v;
}

size_t jg_gcn_norm_coo_workspace_bytes(int64_t n_edges, int64_t n_nodes) {
    if (n_edges < 0 || n_nodes < 0) return 0;
    return carve_norm_coo(nullptr, n_edges, n_nodes).bytes;
}

int jg_gcn_norm_coo(const int32_t* edge_index, const float* w, int64_t n_edges, int64_t n_nodes, float fill,
                    int add_self_loops, int32_t* out_src, int32_t* out_dst, float* out_w, int64_t* out_count,
                    void* workspace, size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(n_edges >= 0 && n_nodes >= 0, JG_EINVAL, "gcn_norm_coo: negative size");
    JG_CHECK_ARG(out_count, JG_EINVAL, "gcn_norm_coo: null count");
    JG_CHECK_ARG(n_edges + n_nodes == 0 || (out_src && out_dst && out_w), JG_EINVAL, "gcn_norm_coo: null output");
    JG_CHECK_ARG(n_edges == 0 || edge_index, JG_EINVAL, "gcn_norm_coo: null edge_index");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_gcn_norm_coo_workspace_bytes(n_edges, n_nodes), JG_EWORKSPACE,
                 "gcn_norm_coo: workspace %zu < %zu", workspace_bytes, jg_gcn_norm_coo_workspace_bytes(n_edges, n_nodes));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    NormCooWs nw = carve_norm_coo(workspace, n_edges, n_nodes);
    // degrees come from the destination-major order (sums in list order, by a fixed tree beyond kLongColumn entries); its
    // arrays are scratch here
    int rc = jg_gcn_norm_compressed(edge_index, w, n_edges, n_nodes, fill, add_self_loops, 0, nw.tmp_idx, nw.tmp_off,
                                    nw.tmp_w, nullptr, nullptr, nullptr, out_count, nw.convert, nw.convert_bytes, stream);
    if (rc != JG_OK) return rc;
    ConvertWs ws = carve_convert(nw.convert, n_edges + n_nodes, n_nodes);  // dis, loop_w and kept live there
    const bool unit = (w == nullptr) && fill == 1.0f;
    if (!add_self_loops) {   // the list as given, every weight scaled by the two degrees
        if (n_edges > 0) {
            norm_coo_plain_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(edge_index, edge_index + n_edges, w, ws.dis,
                                                                            n_edges, out_src, out_dst, out_w);
            JG_LAUNCH_CHECK();
        }
        return JG_OK;
    }
    if (n_edges > 0) {
        keep_flags_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(edge_index, edge_index + n_edges, n_edges, nw.pos);
        JG_LAUNCH_CHECK();
        rc = exclusive_scan(nw.pos, nw.pos, n_edges, nw.pos_sums, st);
        if (rc != JG_OK) return rc;
    }
    if (n_edges + n_nodes > 0) {
        write_norm_coo_kernel<<<blocks_for(n_edges + n_nodes, 256), 256, 0, st>>>(
            edge_index, edge_index + n_edges, w, unit ? nullptr : ws.loop_w, nw.pos, ws.dis, n_edges, n_nodes, ws.kept,
            out_src, out_dst, out_w);
        JG_LAUNCH_CHECK();
    }
    return JG_OK;
}


size_t jg_partition_split_workspace_bytes(int64_t nnz) {
    if (nnz < 0) return 0;
    Carver c(nullptr);
    c.take<int>(nnz + 1);
    c.take<int>(scan_temp_ints(nnz + 1));
    return c.total();
}

int jg_partition_split(const int32_t* idx, const int32_t* off, const float* w, int64_t n_rows, int64_t nnz, int32_t lo,
                       int32_t hi, int32_t* int_idx, int32_t* int_off, float* int_w, int32_t* halo_idx,
                       int32_t* halo_off, float* halo_w, int64_t* out_counts, void* workspace, size_t workspace_bytes,
                       jg_stream_t stream) {
    JG_CHECK_ARG(n_rows >= 0 && nnz >= 0 && lo <= hi, JG_EINVAL, "partition_split: bad sizes");
    JG_CHECK_ARG(off && int_off && halo_off && out_counts, JG_EINVAL, "partition_split: null offsets/counts");
    JG_CHECK_ARG(nnz == 0 || (idx && w && int_idx && int_w && halo_idx && halo_w), JG_EINVAL, "partition_split: null array");
    JG_CHECK_ARG(nnz < INT32_MAX && n_rows < INT32_MAX, JG_ESHAPE, "partition_split: sizes beyond int32");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_partition_split_workspace_bytes(nnz), JG_EWORKSPACE,
                 "partition_split: workspace too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Carver c(workspace);
    int* pos = c.take<int>(nnz + 1);
    int* sums = c.take<int>(scan_temp_ints(nnz + 1));
    interior_flags_kernel<<<blocks_for(nnz + 1, 256), 256, 0, st>>>(idx, nnz, lo, hi, pos);
    JG_LAUNCH_CHECK();
    int rc = exclusive_scan(pos, pos, nnz + 1, sums, st);
    if (rc != JG_OK) return rc;
    if (nnz > 0) {
        split_write_kernel<<<blocks_for(nnz, 256), 256, 0, st>>>(idx, w, pos, nnz, lo, hi, int_idx, int_w, halo_idx, halo_w);
        JG_LAUNCH_CHECK();
    }
    split_offsets_kernel<<<blocks_for(n_rows + 1, 256), 256, 0, st>>>(off, pos, n_rows, int_off, halo_off, out_counts);
    JG_LAUNCH_CHECK();
    return JG_OK;
}


struct UndirectedWs {
    void* convert;
    size_t convert_bytes;
    int32_t* idx;
    float* w;
    int* pos;
    int* pos_sums;
    size_t bytes;
};

static UndirectedWs carve_undirected(void* ws, int64_t n_edges, int64_t n_nodes) {
    Carver c(ws);
    UndirectedWs v;
    v.convert_bytes = jg_convert_workspace_bytes(2 * n_edges, n_nodes);
    v.convert = c.take<unsigned char>(v.convert_bytes);
    v.idx = c.take<int32_t>(2 * n_edges + 1);
    v.w = c.take<float>(2 * n_edges + 1);
    v.pos = c.take<int>(2 * n_edges + 1);
    v.pos_sums = c.take<int>(scan_temp_ints(2 * n_edges + 1));
    v.bytes = c.total();
    return v;
}

size_t jg_to_undirected_workspace_bytes(int64_t n_edges, int64_t n_nodes) {
    if (n_edges < 0 || n_nodes < 0) return 0;
    return carve_undirected(nullptr, n_edges, n_nodes).bytes;
}

int jg_to_undirected(const int32_t* edge_index, const float* attr, int64_t n_edges, int64_t n_nodes, int32_t* out_src,
                     int32_t* out_dst, float* out_attr, int64_t* out_count, void* workspace, size_t workspace_bytes,
                     jg_stream_t stream) {
    JG_CHECK_ARG(n_edges >= 0 && n_nodes >= 0, JG_EINVAL, "to_undirected: negative size");
    JG_CHECK_ARG(out_count, JG_EINVAL, "to_undirected: null count");
    JG_CHECK_ARG(n_edges == 0 || (edge_index && out_src && out_dst && out_attr), JG_EINVAL, "to_undirected: null array");
    JG_CHECK_ARG(2 * n_edges <= INT32_MAX - 1 && n_nodes < INT32_MAX, JG_ESHAPE, "to_undirected: sizes beyond int32");
    JG_CHECK_ARG(workspace && workspace_bytes >= jg_to_undirected_workspace_bytes(n_edges, n_nodes), JG_EWORKSPACE,
                 "to_undirected: workspace too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t m = 2 * n_edges;
    UndirectedWs uw = carve_undirected(workspace, n_edges, n_nodes);
    ConvertWs ws = carve_convert(uw.convert, m + n_nodes, n_nodes);
    SortSrc first = {};
    first.mode = 2;
    first.coo_src = edge_index;
    first.coo_dst = edge_index + n_edges;
    first.coo_w = attr;
    first.count = m;
    int32_t* skey = nullptr;
    int rc = radix_sort(first, n_nodes, 1, nullptr, ws, uw.idx, uw.w, &skey, st);   // by (row, col), stable
    if (rc != JG_OK) return rc;
    first_of_run_kernel<<<blocks_for(m + 1, 256), 256, 0, st>>>(skey, uw.idx, m, uw.pos);
    JG_LAUNCH_CHECK();
    rc = exclusive_scan(uw.pos, uw.pos, m + 1, uw.pos_sums, st);
    if (rc != JG_OK) return rc;
    compact_runs_kernel<<<blocks_for(m + 1, 256), 256, 0, st>>>(skey, uw.idx, uw.w, uw.pos, m, out_src, out_dst, out_attr,
                                                                 out_count);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

}  // extern "C"
