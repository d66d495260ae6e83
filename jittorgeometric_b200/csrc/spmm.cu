// Weighted segment aggregation (CSC forward / CSR backward SpMM) for sm_100a.
//
//   out[v,:] = sum_{j in [off[v], off[v+1])} w[j] * x[idx[j],:]
//
// Replaces the reference's AggregateOp (ops/cpp/aggregate_op.cc:26-105) and the
// cuSPARSE SpMM behind SpmmCsr/SpmmCoo (ops/spmmcsr.py:31, ops/spmmcoo.py:34).
//
// Work decomposition.  A "work id" is either one piece (<= chunk entries) of a
// hub row listed in the plan, or one ordinary row.  A persistent grid of warps
// pulls tickets from a global counter, hub pieces first, so the longest items
// start earliest; a ticket is one to eight ids, fewer the less work there is.
// Who walks an id depends on the width:
//   F <= 31            aggregate_narrow_kernel: 4 to 32 lanes a row, rows side by side
//   F = 32, 36 .. 64   aggregate_stream_kernel, or row by row where that is faster
//   F = 68 .. 512      aggregate_rows_kernel: a warp a row, 128-bit gathers
//   any other          aggregate_any_kernel: scalar loads along the columns
// Indices and weights are read 32 at a time, coalesced, ahead of their use; the
// last three stage them in shared memory or hand them round with shuffles.  The
// kernels are sensitive to instruction issue as well as to memory latency.
// Memory-bound: per nonzero one 4 B index, one 4 B weight and one F*4 B row.
//
// Determinism.  Each output row is produced by exactly one warp (or, for a hub
// row, by a fixed-order sum of its pieces' partial rows held in scratch), so
// results do not depend on which warp ran which id.  No atomics touch data; the
// only atomic is the ticket counter.
#include "common.cuh"

namespace jg {

// The kernels walk entries by 32-bit positions in steps of 32, the streaming one two windows ahead of a ticket padded to
// whole steps: beyond this a position would wrap before it reaches the end.
constexpr int64_t kMaxEntries = INT32_MAX - 128;

struct PlanHeader {
    int32_t n_hubs;
    int32_t n_items;
    int32_t chunk;
    int32_t max_hubs;
    int32_t max_items;
    int32_t pad[3];
};

struct PlanView {
    PlanHeader* hdr;
    int32_t* hub_row;    // [max_hubs] row id of each hub
    int32_t* hub_first;  // [max_hubs] first partial slot of each hub
    int32_t* item_hub;   // [max_items] hub index of each piece
    int32_t* item_k;     // [max_items] piece number within its hub
};

static inline int64_t plan_max_hubs(int64_t nnz, int32_t chunk) { return nnz / ((int64_t)chunk + 1) + 1; }
static inline int64_t plan_max_items(int64_t nnz, int32_t chunk) {
    return nnz / chunk + plan_max_hubs(nnz, chunk) + 1;
}

static PlanView plan_view(void* plan, int64_t nnz, int32_t chunk, size_t* bytes) {
    Carver c(plan);
    PlanView v;
    v.hdr = c.take<PlanHeader>(1);
    v.hub_row = c.take<int32_t>(plan_max_hubs(nnz, chunk));
    v.hub_first = c.take<int32_t>(plan_max_hubs(nnz, chunk));
    v.item_hub = c.take<int32_t>(plan_max_items(nnz, chunk));
    v.item_k = c.take<int32_t>(plan_max_items(nnz, chunk));
    if (bytes) *bytes = c.total();
    return v;
}

__global__ void plan_header_kernel(PlanHeader* hdr, PlanHeader h) { *hdr = h; }

__global__ void plan_build_kernel(const int32_t* __restrict__ off, int64_t n, PlanView p, int32_t chunk) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        int32_t deg = off[v + 1] - off[v];
        if (deg > chunk) {
            int32_t pieces = (deg + chunk - 1) / chunk;
            int32_t h = atomicAdd(&p.hdr->n_hubs, 1);
            int32_t first = atomicAdd(&p.hdr->n_items, pieces);
            p.hub_row[h] = (int32_t)v;
            p.hub_first[h] = first;
            for (int32_t k = 0; k < pieces; k++) {
                p.item_hub[first + k] = h;
                p.item_k[first + k] = k;
            }
        }
    }
}

constexpr int kGrab = 8;      // most work ids taken per ticket (AggArgs::grab: fewer when the work is short)
constexpr int kBlock = 256;   // threads per CTA

struct AggArgs {
    float* out;
    const float* x;
    const int32_t* idx;
    const int32_t* off;
    const float* w;
    int64_t n_out;
    int64_t f;
    const PlanHeader* hdr;  // null: no plan
    const int32_t* hub_row;
    const int32_t* hub_first;
    const int32_t* item_hub;
    const int32_t* item_k;
    float* partial;
    unsigned long long* ticket;
    int accumulate;  // 1: add the aggregated row to what `out` already holds (old + sum)
    int64_t max_items;  // host-side upper bound on the plan's pieces (sizes the grid)
    int64_t n_in, nnz;  // rows of x and entries (choose the kernel)
    const float* bias;  // epilogue on finished output rows: + bias[column] (null: none) ...
    const float* addend;  // [n_out, f] combined with the sum before the bias (null: none): scale * sum + add_scale * addend
    float scale, add_scale;
    int relu;           // ... then max(., 0)
    int ordered;        // 1: every row must be summed in stored order (no lane groups taking alternate entries)
    int reserve_ctas;   // CTA slots of the persistent grid left free for a kernel that runs beside this one
    int grab;           // work ids per ticket, 1..kGrab (set by the launcher from the amount of work)
};


// Exact mode rounds multiply and add separately, as the reference CPU loop does (scalar instructions: the packed
// pair of mul.rn and add.rn comes back fused); the fused mode uses one FMA per term, two terms per instruction -
// at the widths that use it the kernels are bound by instruction issue, and a packed FMA rounds as two scalar ones.
__device__ __forceinline__ void fma_pair(float& a0, float& a1, float v0, float v1, unsigned long long ww) {
    unsigned long long a, v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(v0), "f"(v1));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(v), "l"(ww));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
}
template <bool EXACT>
__device__ __forceinline__ void axpy4(float4& a, const float4& v, float w) {
    if (EXACT) {
        a.x = __fadd_rn(__fmul_rn(v.x, w), a.x);
        a.y = __fadd_rn(__fmul_rn(v.y, w), a.y);
        a.z = __fadd_rn(__fmul_rn(v.z, w), a.z);
        a.w = __fadd_rn(__fmul_rn(v.w, w), a.w);
    } else {
        unsigned long long ww;
        asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w));
        fma_pair(a.x, a.y, v.x, v.y, ww);
        fma_pair(a.z, a.w, v.z, v.w, ww);
    }
}

// Epilogue of a finished output element: scale * sum + add_scale * addend, + bias, ReLU (each if asked for).
// `h`: the addend's element.
__device__ __forceinline__ float finish_with(const AggArgs& a, float v, float h, int64_t col) {
    if (a.addend) v = fmaf(a.scale, v, __fmul_rn(a.add_scale, h));
    if (a.bias) v += __ldg(a.bias + col);
    if (a.relu) v = fmaxf(v, 0.f);
    return v;
}
__device__ __forceinline__ float finish_value(const AggArgs& a, float v, size_t at, int64_t col) {
    return finish_with(a, v, a.addend ? __ldg(a.addend + at) : 0.f, col);
}
// What a kernel instantiation compiles in: nothing, bias and ReLU, or the sum with the addend.
enum Epilogue { kPlain = 0, kBiasAct = 1, kCombine = 2 };
template <int EPI>
__device__ __forceinline__ float4 finish_value4(const AggArgs& a, float4 v, size_t at, int col) {
    if (EPI == kCombine) {
        const float4 h = __ldcs(reinterpret_cast<const float4*>(a.addend + at));
        v.x = fmaf(a.scale, v.x, __fmul_rn(a.add_scale, h.x)); v.y = fmaf(a.scale, v.y, __fmul_rn(a.add_scale, h.y));
        v.z = fmaf(a.scale, v.z, __fmul_rn(a.add_scale, h.z)); v.w = fmaf(a.scale, v.w, __fmul_rn(a.add_scale, h.w));
    }
    if (EPI == kBiasAct) {
        if (a.bias) {
            const float4 b4 = __ldg(reinterpret_cast<const float4*>(a.bias + col));
            v.x += b4.x; v.y += b4.y; v.z += b4.z; v.w += b4.w;
        }
        if (a.relu) {
            v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
        }
    }
    return v;
}

// Row-by-row kernel (F <= 4*G*VPL).  G lanes cover one feature row, 32/G entries are gathered side by side (one "step"),
// B steps per batch.  G = 32, all widths above 64: entries are added in stored order.  G = 8 and 16, the widths up to 64
// where the streaming kernel below loses (see the dispatch): the lane groups' sums are added at the end.
// EPI compiles in an epilogue (instantiations of their own: the registers of one cost the others 3 %).
// FULL: the row is exactly 4*G*VPL floats wide (everything about the width folds at compile time).
// !FULL: any 16-byte-aligned width up to that; lanes whose columns lie beyond it sit out.
template <int G, int VPL, int B, int MINB, int EPI, bool FULL>
__global__ void __launch_bounds__(kBlock, MINB) aggregate_rows_kernel(AggArgs a) {
    constexpr int EPS = 32 / G;
    constexpr bool EXACT = G == 32;
    const int F = FULL ? 4 * G * VPL : (int)a.f;
    __shared__ int2 s_tile[kBlock / 32][32];
    const int lane = lane_id();
    const int sub = lane / G;
    const int fl = lane % G;
    bool qok[VPL];
#pragma unroll
    for (int q = 0; q < VPL; q++) qok[q] = FULL || (fl + q * G) * 4 < F;
    int2* tile = s_tile[threadIdx.x / 32];
    const char* xb = reinterpret_cast<const char*>(a.x) + fl * 16;
    const int64_t n_items = a.hdr ? a.hdr->n_items : 0;
    const int chunk = a.hdr ? a.hdr->chunk : 0x7fffffff;
    const int64_t total = n_items + a.n_out;
    const int grab = a.grab;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.ticket, (unsigned long long)grab);
        base = __shfl_sync(kFull, base, 0);
        if ((int64_t)base >= total) break;
        const int64_t row0 = (int64_t)base - n_items;
        int32_t offv = 0;
        {
            const int64_t r = row0 + lane;
            if (lane <= grab && r >= 0 && r <= a.n_out) offv = a.off[r];
        }
        int32_t pf_pos = -1;  // position of the prefetched tile
        int32_t pf_lim = -1;  // ... which holds entries below this bound only
        int pf_idx = 0;
        float pf_w = 0.f;
#pragma unroll 1
        for (int i = 0; i < grab; i++) {
            const int64_t id = (int64_t)base + i;
            if (id >= total) break;
            int32_t s, e, lim;
            float* dst;
            const bool add_old = a.accumulate && id >= n_items;
            if (id < n_items) {
                const int h = a.item_hub[id];
                const int k = a.item_k[id];
                const int row = a.hub_row[h];
                const int32_t rs = a.off[row], re = a.off[row + 1];
                s = rs + k * chunk;
                e = min(re, s + chunk);
                lim = re;  // the next piece of the same hub continues where this one ends
                dst = a.partial + (size_t)(a.hub_first[h] + k) * F;
            } else {
                s = __shfl_sync(kFull, offv, i);
                e = __shfl_sync(kFull, offv, i + 1);
                if (e - s > chunk) continue;  // hub row: its pieces are separate work ids
                // entries of the following rows of this grab are contiguous with this row's
                const int64_t left = a.n_out - row0;
                const int last = left < grab ? (int)left : grab;
                lim = __shfl_sync(kFull, offv, last);
                dst = a.out + (size_t)(id - n_items) * F;
            }
            if (lim != pf_lim) pf_pos = -1;  // a tile prefetched under another bound is not reusable
            pf_lim = lim;
            float4 acc[VPL];
#pragma unroll
            for (int q = 0; q < VPL; q++) acc[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int32_t j0 = s; j0 < e; j0 += 32) {
                int cur_idx = pf_idx;
                float cur_w = pf_w;
                if (pf_pos != j0) {
                    cur_idx = 0;
                    cur_w = 0.f;
                    if (j0 + lane < lim) {
                        cur_idx = ld_stream(a.idx + j0 + lane);
                        cur_w = ld_stream(a.w + j0 + lane);
                    }
                }
                // next tile: the rest of this row, or the start of the next row of the grab
                pf_pos = min(j0 + 32, e);
                pf_idx = 0;
                pf_w = 0.f;
                if (pf_pos + lane < lim) {
                    pf_idx = ld_stream(a.idx + pf_pos + lane);
                    pf_w = ld_stream(a.w + pf_pos + lane);
                }
                __syncwarp();
                tile[lane] = make_int2(cur_idx, __float_as_int(cur_w));
                __syncwarp();
                const int cnt = min(32, e - j0);
                int t = 0;
                for (; t + EPS * B <= cnt; t += EPS * B) {  // full batches: no predicates
                    float4 v[B][VPL];
                    float wv[B];
#pragma unroll
                    for (int u = 0; u < B; u++) {
                        const int2 p = tile[t + u * EPS + sub];
                        wv[u] = __int_as_float(p.y);
                        const float4* g = reinterpret_cast<const float4*>(xb + (size_t)(unsigned)p.x * (size_t)(F * 4));
#pragma unroll
                        for (int q = 0; q < VPL; q++) v[u][q] = qok[q] ? __ldg(g + q * G) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int u = 0; u < B; u++)
#pragma unroll
                        for (int q = 0; q < VPL; q++) axpy4<EXACT>(acc[q], v[u][q], wv[u]);
                }
                if (t < cnt) {  // last, partial batch
                    // Four entries per step: steps that lie wholly beyond the row are skipped by a warp-uniform test (most
                    // rows of a power-law graph are shorter than one step; 32 columns: -6 % time).  With one or two
                    // entries per step the test measured 5 % slower, it breaks up the batch of loads.
                    float4 v[B][VPL];
                    float wv[B];
#pragma unroll
                    for (int u = 0; u < B; u++) {
                        const int k = t + u * EPS + sub;
                        wv[u] = 0.f;
#pragma unroll
                        for (int q = 0; q < VPL; q++) v[u][q] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if ((EPS < 4 || t + u * EPS < cnt) && k < cnt) {
                            const int2 p = tile[k];
                            wv[u] = __int_as_float(p.y);
                            const float4* g = reinterpret_cast<const float4*>(xb + (size_t)(unsigned)p.x * (size_t)(F * 4));
#pragma unroll
                            for (int q = 0; q < VPL; q++)
                                if (qok[q]) v[u][q] = __ldg(g + q * G);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < B; u++) {
                        if (EPS < 4 || t + u * EPS < cnt) {
#pragma unroll
                            for (int q = 0; q < VPL; q++) axpy4<EXACT>(acc[q], v[u][q], wv[u]);
                        }
                    }
                }
            }
#pragma unroll
            for (int o = G; o < 32; o <<= 1)
#pragma unroll
                for (int q = 0; q < VPL; q++) {
                    acc[q].x += __shfl_xor_sync(kFull, acc[q].x, o);
                    acc[q].y += __shfl_xor_sync(kFull, acc[q].y, o);
                    acc[q].z += __shfl_xor_sync(kFull, acc[q].z, o);
                    acc[q].w += __shfl_xor_sync(kFull, acc[q].w, o);
                }
            if (sub == 0) {
                float4* o = reinterpret_cast<float4*>(dst) + fl;
#pragma unroll
                for (int q = 0; q < VPL; q++) {
                    if (!qok[q]) continue;
                    if (add_old) {
                        const float4 old = o[q * G];
                        acc[q].x = __fadd_rn(old.x, acc[q].x);
                        acc[q].y = __fadd_rn(old.y, acc[q].y);
                        acc[q].z = __fadd_rn(old.z, acc[q].z);
                        acc[q].w = __fadd_rn(old.w, acc[q].w);
                    }
                    if (EPI != kPlain && id >= n_items)   // a finished output row (pieces of hub rows get theirs in the fix-up)
                        acc[q] = finish_value4<EPI>(a, acc[q], (size_t)(id - n_items) * F + 4 * (fl + q * G), 4 * (fl + q * G));
                    __stcs(o + q * G, acc[q]);
                }
            }
        }
    }
}

// Streaming kernel of the widths up to 64.  G lanes (8 or 16) cover one feature row of F = 32 or 36 to 64 floats, 32/G
// entries of a row are gathered side by side (one "step").  EPI compiles in the epilogue (a separate
// instantiation, so the plain kernel is untouched).  The width is a template parameter: with it in a register the
// 40-column form was slower than the 64-column one.
//
// The segments of a ticket (a piece of a hub row, or up to eight rows) are walked as ONE stream of entries, each segment
// padded to whole steps: a window of 32 stream positions at a time is looked up by the lanes (position -> segment by a
// search over the ticket's prefix lengths), staged in shared memory as (index, weight) pairs and marked where a
// segment ends.  Batches of B steps are double-buffered in registers across row ends, so the gathers of the next
// rows are in flight while a row is summed and stored; walked row by row, a row of a dozen entries cost two or
// three exposed memory latencies.  The next ticket, and its segments' bounds, are fetched while this one is walked.
// At 64 registers (four CTAs per SM) the plain and the combining form spill 32 bytes at 36 to 60 columns, the bias form 80,
// both epilogues 80 at 64 columns, none at 32.
template <int F, int B, int MINB, int EPI>
__global__ void __launch_bounds__(kBlock, MINB) aggregate_stream_kernel(AggArgs a) {
    constexpr int G = F <= 32 ? 8 : 16;
    constexpr int EPS = 32 / G;
    constexpr int NBW = 32 / (EPS * B);      // batches per window of 32 stream positions
    static_assert(F % 4 == 0 && F <= 4 * G && NBW >= 1 && NBW * EPS * B == 32, "a window holds whole batches");
    static_assert(kGrab <= 8, "the segment search takes three steps");
    __shared__ int2 s_tile[kBlock / 32][2][32];
    const int lane = lane_id();
    const int sub = lane / G;
    const int fl = lane % G;
    const bool mine = fl * 4 < F;    // this lane holds columns of a row
    int2(*tile)[32] = s_tile[threadIdx.x / 32];
    const char* xb = reinterpret_cast<const char*>(a.x) + fl * 16;
    const int64_t n_items = a.hdr ? a.hdr->n_items : 0;
    const int chunk = a.hdr ? a.hdr->chunk : 0x7fffffff;
    const int grab = a.grab;
    // a piece of a hub is a ticket of its own (with four of them in one warp a small graph's tail was longer than its
    // work: 50 k rows, 1.3 M entries, 36 columns, both directions 0.20 ms, 0.12 row by row), rows come `grab` at a time
    const int64_t tickets = n_items + (a.n_out + grab - 1) / grab;
    auto first_id = [&](int64_t ticket) { return ticket < n_items ? ticket : n_items + (ticket - n_items) * grab; };

    // lane i's segment of the ticket: first entry and length (-1: none, a hub row is walked as pieces)
    auto load_segments = [&](int64_t ticket, int& s, int& len) {
        s = 0; len = -1;
        const int64_t id = first_id(ticket) + lane;
        if (lane < (ticket < n_items ? 1 : grab) && id < n_items + a.n_out) {
            if (id < n_items) {
                const int h = a.item_hub[id], k = a.item_k[id];
                const int row = a.hub_row[h];
                s = a.off[row] + k * chunk;
                len = min(a.off[row + 1] - s, chunk);
            } else {
                const int64_t row = id - n_items;
                s = a.off[row];
                len = a.off[row + 1] - s;
                if (len > chunk) len = -1;
            }
        }
    };
    auto take = [&]() -> unsigned long long { return lane == 0 ? atomicAdd(a.ticket, 1ull) : 0ull; };

    int64_t ticket = (int64_t)__shfl_sync(kFull, take(), 0);
    if (ticket >= tickets) return;
    int seg_s, seg_len;
    load_segments(ticket, seg_s, seg_len);
    unsigned long long coming = take();
    for (;;) {
        const int64_t base = first_id(ticket);
        const int64_t next_ticket = (int64_t)__shfl_sync(kFull, coming, 0);
        int nxt_s, nxt_len;
        load_segments(next_ticket, nxt_s, nxt_len);
        if (next_ticket < tickets) coming = take();

        const int padded = seg_len > 0 ? (seg_len + EPS - 1) / EPS * EPS : 0;
        int incl = padded;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        const int T = __shfl_sync(kFull, incl, 7);
        const int excl = incl - padded;
        unsigned todo = __ballot_sync(kFull, seg_len > 0);

        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        // stores segment `seg` and clears the accumulators
        auto flush = [&](int seg) {
            const int64_t id = base + seg;
            const bool row = id >= n_items;     // else a piece: its partial row, finished by the fix-up
#pragma unroll
            for (int o = G; o < 32; o <<= 1) {
                acc.x += __shfl_xor_sync(kFull, acc.x, o);
                acc.y += __shfl_xor_sync(kFull, acc.y, o);
                acc.z += __shfl_xor_sync(kFull, acc.z, o);
                acc.w += __shfl_xor_sync(kFull, acc.w, o);
            }
            if (sub == 0 && mine) {
                float4* o = reinterpret_cast<float4*>(row ? a.out + (size_t)(id - n_items) * F
                                                          : a.partial + (size_t)(a.hub_first[a.item_hub[id]] + a.item_k[id]) * F) + fl;
                if (row && a.accumulate) {
                    const float4 old = *o;
                    acc.x = __fadd_rn(old.x, acc.x);
                    acc.y = __fadd_rn(old.y, acc.y);
                    acc.z = __fadd_rn(old.z, acc.z);
                    acc.w = __fadd_rn(old.w, acc.w);
                }
                if (EPI != kPlain && row) acc = finish_value4<EPI>(a, acc, (size_t)(id - n_items) * F + 4 * fl, 4 * fl);
                __stcs(o, acc);
            }
            acc = make_float4(0.f, 0.f, 0.f, 0.f);
        };
        for (unsigned empty = __ballot_sync(kFull, seg_len == 0); empty; empty &= empty - 1) flush(__ffs(empty) - 1);

        if (T > 0) {
            int pf_idx, pf_w;
            bool pf_last;
            // this lane's position of the window that starts at p0
            auto fetch = [&](int p0) {
                const int p = p0 + lane;
                pf_idx = -1; pf_w = 0; pf_last = false;
                if (p0 >= T) return;
                int g = 0;
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    if (p >= __shfl_sync(kFull, incl, g + o - 1)) g += o;
                const int q = p - __shfl_sync(kFull, excl, g);
                const int len = __shfl_sync(kFull, seg_len, g), s = __shfl_sync(kFull, seg_s, g);
                const int pad = __shfl_sync(kFull, padded, g);
                if (p < T) {
                    if (q < len) {
                        pf_idx = ld_stream(a.idx + s + q);
                        pf_w = __float_as_int(ld_stream(a.w + s + q));
                    }
                    pf_last = q == pad - 1;
                }
            };
            unsigned ends0 = 0, ends1 = 0;    // window positions that end a segment, by window parity
            auto stage = [&](int window) {
                __syncwarp();
                tile[window & 1][lane] = make_int2(pf_idx, pf_w);
                const unsigned m = __ballot_sync(kFull, pf_last);
                if (window & 1) ends1 = m; else ends0 = m;
                __syncwarp();
                fetch(32 * (window + 1));
            };
            auto issue = [&](float4 (&v)[B], int bi) {
                const int2* t = tile[(bi / NBW) & 1] + (bi % NBW) * (B * EPS) + sub;
#pragma unroll
                for (int u = 0; u < B; u++) {
                    const int src = t[u * EPS].x;
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (src >= 0 && mine) v[u] = __ldg(reinterpret_cast<const float4*>(xb + (size_t)(unsigned)src * (size_t)(F * 4)));
                }
            };
            auto consume = [&](float4 (&v)[B], int bi) {
                const int w = bi / NBW, first = (bi % NBW) * (B * EPS);
                const int2* t = tile[w & 1] + first + sub;
                const unsigned ends = ((w & 1) ? ends1 : ends0) >> first;
#pragma unroll
                for (int u = 0; u < B; u++) {
                    axpy4<false>(acc, v[u], __int_as_float(t[u * EPS].y));
                    if ((ends >> (u * EPS)) & ((1u << EPS) - 1u)) {
                        flush(__ffs(todo) - 1);
                        todo &= todo - 1;
                    }
                }
            };
            const int n_batches = (T + B * EPS - 1) / (B * EPS);
            float4 v0[B], v1[B];
            fetch(0);
            stage(0);
            issue(v0, 0);
            for (int bi = 0; bi < n_batches; bi += 2) {
                if (bi + 1 < n_batches) {
                    if ((bi + 1) % NBW == 0) stage((bi + 1) / NBW);
                    issue(v1, bi + 1);
                }
                consume(v0, bi);
                if (bi + 1 >= n_batches) break;
                if (bi + 2 < n_batches) {
                    if ((bi + 2) % NBW == 0) stage((bi + 2) / NBW);
                    issue(v0, bi + 2);
                }
                consume(v1, bi + 1);
            }
        }
        if (next_ticket >= tickets) break;
        ticket = next_ticket;
        seg_s = nxt_s; seg_len = nxt_len;
    }
}

// Any feature width: lanes stride over columns with scalar loads, up to 256 columns per sweep.
template <int Q>
__device__ __forceinline__ void warp_segment_any(const AggArgs& a, int32_t s, int32_t e, float* dst, bool add_old, bool final_row) {
    constexpr int UNROLL = Q <= 2 ? 8 : 4;
    const int lane = lane_id();
    const int64_t F = a.f;
    for (int64_t c0 = 0; c0 < F; c0 += 32 * Q) {
        float acc[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) acc[q] = 0.f;
        for (int32_t j0 = s; j0 < e; j0 += 32) {
            const int cnt = min(32, e - j0);
            int cur_idx = 0;
            float cur_w = 0.f;
            if (j0 + lane < e) {
                cur_idx = ld_stream(a.idx + j0 + lane);
                cur_w = ld_stream(a.w + j0 + lane);
            }
            for (int t = 0; t < cnt; t += UNROLL) {
                float v[UNROLL][Q];
                float wv[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; u++) {
                    const int k = t + u;
                    const int src = __shfl_sync(kFull, cur_idx, k & 31);
                    wv[u] = __shfl_sync(kFull, cur_w, k & 31);
                    const float* p = a.x + (size_t)src * F + c0 + lane;
#pragma unroll
                    for (int q = 0; q < Q; q++)
                        v[u][q] = (k < cnt && c0 + q * 32 + lane < F) ? __ldg(p + q * 32) : 0.f;
                    if (k >= cnt) wv[u] = 0.f;
                }
#pragma unroll
                for (int u = 0; u < UNROLL; u++)
#pragma unroll
                    for (int q = 0; q < Q; q++) acc[q] = __fadd_rn(__fmul_rn(v[u][q], wv[u]), acc[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (c0 + q * 32 + lane < F) {
                float v = add_old ? __fadd_rn(dst[c0 + q * 32 + lane], acc[q]) : acc[q];
                const int64_t col = c0 + q * 32 + lane;
                if (final_row) v = finish_value(a, v, (size_t)(dst - a.out) + col, col);
                dst[col] = v;
            }
    }
}

// Any feature width: one warp per work id, column-strided scalar loads, Q * 32 columns per sweep
// (Q = 2 or 4 for widths up to 64 or 128, so that narrow odd widths do not pay for empty sweeps).
template <int Q>
__global__ void __launch_bounds__(kBlock) aggregate_any_kernel(AggArgs a) {
    const int lane = lane_id();
    const int64_t n_items = a.hdr ? a.hdr->n_items : 0;
    const int chunk = a.hdr ? a.hdr->chunk : 0x7fffffff;
    const int64_t total = n_items + a.n_out;
    const int64_t F = a.f;
    const int grab = a.grab;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.ticket, (unsigned long long)grab);
        base = __shfl_sync(kFull, base, 0);
        if ((int64_t)base >= total) break;
        // offsets of up to kGrab consecutive ordinary rows with one coalesced read
        const int64_t row0 = (int64_t)base - n_items;
        int32_t offv = 0;
        {
            const int64_t r = row0 + lane;
            if (lane <= grab && r >= 0 && r <= a.n_out) offv = a.off[r];
        }
#pragma unroll 1
        for (int i = 0; i < grab; i++) {
            const int64_t id = (int64_t)base + i;
            if (id >= total) break;
            int32_t s, e;
            float* dst;
            if (id < n_items) {
                const int h = a.item_hub[id];
                const int k = a.item_k[id];
                const int row = a.hub_row[h];
                const int32_t rs = a.off[row], re = a.off[row + 1];
                s = rs + k * chunk;
                e = min(re, s + chunk);
                dst = a.partial + (size_t)(a.hub_first[h] + k) * F;
            } else {
                // lane i of this grab holds off[row], lane i+1 holds off[row+1]
                const int64_t row = id - n_items;
                s = __shfl_sync(kFull, offv, i);
                e = __shfl_sync(kFull, offv, i + 1);
                if (e - s > chunk) continue;  // hub row: its pieces are separate work ids
                dst = a.out + (size_t)row * F;
            }
            warp_segment_any<Q>(a, s, e, dst, a.accumulate && id >= n_items, id >= n_items);
        }
    }
}

// Narrow feature widths (F <= G <= 32, any alignment): G lanes own one work id (an output row or a
// piece of a hub row), so 32/G of them are walked side by side, each in its own stored order with
// separately rounded multiply and add - the result of a row is bit-identical to the sequential
// reference loop.  The G lanes fetch G consecutive (index, weight) entries with one coalesced load
// each and hand them round with width-G shuffles; lane c gathers column c of every source row.
// All groups run the trip count of the longest of their segments, with predicates, so the shuffles
// stay convergent.  The last layer of a GCN (a handful of classes) is this shape.
// EPI: an epilogue is asked for (with its tests in the plain form, 14 columns and 10 M entries took 2 % longer).
template <int G, bool EPI>
__global__ void __launch_bounds__(kBlock) aggregate_narrow_kernel(AggArgs a) {
    constexpr int R = 32 / G;          // work ids per warp step
    constexpr int ROUNDS = 4;          // steps per ticket
    const int lane = lane_id();
    const int grp = lane / G, c = lane % G;
    const int64_t n_items = a.hdr ? a.hdr->n_items : 0;
    const int chunk = a.hdr ? a.hdr->chunk : 0x7fffffff;
    const int64_t total = n_items + a.n_out;
    const int F = (int)a.f;
    const bool col_ok = c < F;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.ticket, (unsigned long long)(R * ROUNDS));
        base = __shfl_sync(kFull, base, 0);
        if ((int64_t)base >= total) break;
#pragma unroll 1
        for (int round = 0; round < ROUNDS; round++) {
            const int64_t id = (int64_t)base + round * R + grp;
            int32_t s = 0, e = 0;
            float* dst = nullptr;
            bool final_row = false;
            if (id < total) {
                if (id < n_items) {
                    const int h = a.item_hub[id];
                    const int k = a.item_k[id];
                    const int row = a.hub_row[h];
                    const int32_t rs = a.off[row], re = a.off[row + 1];
                    s = rs + k * chunk;
                    e = min(re, s + chunk);
                    dst = a.partial + (size_t)(a.hub_first[h] + k) * F;
                } else {
                    const int64_t row = id - n_items;
                    s = a.off[row];
                    e = a.off[row + 1];
                    if (e - s > chunk) {   // hub row: its pieces are separate work ids
                        e = s;
                    } else {
                        dst = a.out + (size_t)row * F;
                        final_row = true;
                    }
                }
            }
            // The addend's element travels while the row is summed, and leaves L2 first: x is what is read again.  Four hops
            // over 1 M rows of 16 columns: 2875 us with the load at the row's end, 2280 here, 2240 read once (sum and
            // three passes behind it 2480).
            float h = 0.f;
            if (EPI && a.addend && final_row && col_ok) h = __ldcs(a.addend + (dst - a.out) + c);
            const int len = e - s;
            int maxlen = len;
#pragma unroll
            for (int o = G; o < 32; o <<= 1) maxlen = max(maxlen, __shfl_xor_sync(kFull, maxlen, o));
            if (G < 32 && (int64_t)base + round * R >= total) break;   // warp-uniform: nothing left in this ticket
            float acc = 0.f;
            for (int j = 0; j < maxlen; j += G) {
                int my_idx = 0;
                float my_w = 0.f;
                if (j + c < len) {
                    my_idx = ld_stream(a.idx + s + j + c);
                    my_w = ld_stream(a.w + s + j + c);
                }
#pragma unroll
                for (int k0 = 0; k0 < G; k0 += 4) {
                    float v[4], wv[4];
                    bool ok[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int k = k0 + u;
                        const int src = __shfl_sync(kFull, my_idx, k, G);
                        wv[u] = __shfl_sync(kFull, my_w, k, G);
                        ok[u] = j + k < len;
                        v[u] = 0.f;
                        if (ok[u] && col_ok) v[u] = __ldg(a.x + (size_t)(unsigned)src * F + c);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (ok[u]) acc = __fadd_rn(__fmul_rn(v[u], wv[u]), acc);
                }
            }
            if (dst && col_ok) {
                float v = acc;
                if (final_row) {
                    if (a.accumulate) v = __fadd_rn(dst[c], v);
                    if (EPI) v = finish_with(a, v, h, c);
                }
                dst[c] = v;
            }
        }
    }
}

// Adds the partial rows of every hub and writes the hub's output row.  A block takes a run of hubs: their rows, piece
// counts and first slots are read side by side, then hubs of up to kFewPieces pieces are summed with one thread per
// (hub, column), all pieces in flight, and the others one by one by the whole block, eight warps each adding an eighth
// of the pieces in order and the eighths in order.  With one thread per (hub, column) whatever the pieces, the
// longest hub's chain of loads was the kernel: 17 us beside a 160 us aggregation of 4.9 M entries (70 pieces), 8 us so;
// 128 columns at a time (16 bytes a lane) where the width allows: 256 columns, 126 M entries 207 -> 94 us.
constexpr int kFewPieces = 8;
__global__ void __launch_bounds__(kBlock) hub_fixup_kernel(AggArgs a) {
    __shared__ int s_row[kBlock], s_first[kBlock], s_pieces[kBlock];
    __shared__ float4 s_sum[kBlock / 32][32];
    const int n_hubs = a.hdr->n_hubs;
    const int chunk = a.hdr->chunk;
    const int F = (int)a.f;
    const int lane = lane_id(), warp = threadIdx.x / 32;
    int per_block = (n_hubs + (int)gridDim.x - 1) / (int)gridDim.x;
    if (per_block > kBlock) per_block = kBlock;
    // 16 bytes a lane where every partial row starts on a 16-byte border; a caller's workspace need not
    const int V = F % 4 == 0 && reinterpret_cast<uintptr_t>(a.partial) % 16 == 0 ? 4 : 1;
    for (int64_t h0 = (int64_t)blockIdx.x * per_block; h0 < n_hubs; h0 += (int64_t)gridDim.x * per_block) {
        const int cnt = n_hubs - h0 < per_block ? (int)(n_hubs - h0) : per_block;
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int row = a.hub_row[h0 + threadIdx.x];
            s_row[threadIdx.x] = row;
            s_first[threadIdx.x] = a.hub_first[h0 + threadIdx.x];
            s_pieces[threadIdx.x] = (a.off[row + 1] - a.off[row] + chunk - 1) / chunk;
        }
        __syncthreads();
        const int64_t values = (int64_t)cnt * F;
        for (int64_t t = threadIdx.x; t < values; t += kBlock) {
            const int h = values < INT32_MAX ? (int)t / F : (int)(t / F), c = (int)(t - (int64_t)h * F);
            const int pieces = s_pieces[h];
            if (pieces > kFewPieces) continue;
            const float* p = a.partial + (size_t)s_first[h] * F + c;
            float v[kFewPieces];
#pragma unroll
            for (int k = 0; k < kFewPieces; k++) v[k] = k < pieces ? __ldg(p + (size_t)k * F) : 0.f;
            float acc = v[0];
#pragma unroll
            for (int k = 1; k < kFewPieces; k++)
                if (k < pieces) acc = __fadd_rn(acc, v[k]);
            float* o = a.out + (size_t)s_row[h] * F + c;
            *o = finish_value(a, a.accumulate ? __fadd_rn(*o, acc) : acc, (size_t)s_row[h] * F + c, c);
        }
        for (int h = 0; h < cnt; h++) {
            const int pieces = s_pieces[h];
            if (pieces <= kFewPieces) continue;
            const int per = (pieces + kBlock / 32 - 1) / (kBlock / 32);
            const int k0 = warp * per, k1 = k0 + per < pieces ? k0 + per : pieces;
            for (int c0 = 0; c0 < F; c0 += 32 * V) {
                const int c = c0 + lane * V;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < F) {
                    const float* p = a.partial + (size_t)s_first[h] * F + c;
                    if (V == 4) {
#pragma unroll 4
                        for (int k = k0; k < k1; k++) {
                            const float4 v = __ldg(reinterpret_cast<const float4*>(p + (size_t)k * F));
                            acc.x = __fadd_rn(acc.x, v.x); acc.y = __fadd_rn(acc.y, v.y);
                            acc.z = __fadd_rn(acc.z, v.z); acc.w = __fadd_rn(acc.w, v.w);
                        }
                    } else {
#pragma unroll 4
                        for (int k = k0; k < k1; k++) acc.x = __fadd_rn(acc.x, __ldg(p + (size_t)k * F));
                    }
                }
                s_sum[warp][lane] = acc;
                __syncthreads();
                // one thread per column of the slab: the eighths in order
                const int col = c0 + (int)threadIdx.x;
                if ((int)threadIdx.x < 32 * V && col < F) {
                    const int l = threadIdx.x / V, q = threadIdx.x % V;
                    float sum = reinterpret_cast<const float*>(&s_sum[0][l])[q];
#pragma unroll
                    for (int g = 1; g < kBlock / 32; g++) sum = __fadd_rn(sum, reinterpret_cast<const float*>(&s_sum[g][l])[q]);
                    float* o = a.out + (size_t)s_row[h] * F + col;
                    *o = finish_value(a, a.accumulate ? __fadd_rn(*o, sum) : sum, (size_t)s_row[h] * F + col, col);
                }
                __syncthreads();
            }
        }
    }
}

// Blocks of the fix-up: one for every four hubs that a plan of `nnz` entries could list, four per SM at most.
static unsigned fixup_blocks(int64_t nnz, int32_t chunk) {
    const int64_t blocks = (plan_max_hubs(nnz, chunk) + 3) / 4, most = (int64_t)sm_count() * 4;
    return (unsigned)(blocks < most ? blocks : most);
}

// Persistent grid: as many CTAs as fit on the device, but no more than the work can feed.  Every warp
// takes at least one ticket (an atomic on one address) to learn that nothing is left, so on a small
// graph a full grid of some ten thousand warps would spend its time queueing on that counter.
template <class K>
static int launch_persistent(K kern, int* blocks_per_sm, const AggArgs& a, cudaStream_t st, int low_grab = 1) {
    if (*blocks_per_sm == 0) {
        int b = 0;
        JG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, kBlock, 0));
        *blocks_per_sm = b > 0 ? b : 1;
    }
    int64_t full = (int64_t)sm_count() * *blocks_per_sm;
    if (a.reserve_ctas > 0) full = full - a.reserve_ctas > sm_count() ? full - a.reserve_ctas : sm_count();
    // Tickets of eight ids keep the atomic rare on a large graph; when a warp would see fewer than about
    // two dozen tickets the tail (the last warps still walking their eight rows while the rest of the
    // device idles) dominates, so the tickets get smaller: a shard of 262 k rows ran at half the per-entry
    // speed of the whole graph with eight ids per ticket.
    AggArgs b = a;
    const int64_t ids = a.n_out + a.max_items;
    int64_t g = ids / (full * (kBlock / 32) * 24);
    // A kernel that pays per ticket (the streaming one: look-ups, an open pipeline) takes up to `low_grab` ids at once
    // as long as that leaves every warp six tickets.
    int64_t low = ids / (full * (kBlock / 32) * 6);
    if (low > low_grab) low = low_grab;
    if (g < low) g = low;
    b.grab = g < 1 ? 1 : (g > kGrab ? kGrab : (int)g);
    const int64_t grabs = low_grab > 1 ? a.max_items + (a.n_out + b.grab - 1) / b.grab     // a piece is a ticket of its own there
                                       : (ids + b.grab - 1) / b.grab;
    int64_t blocks = (grabs + kBlock / 32 - 1) / (kBlock / 32);
    if (blocks > full) blocks = full;
    if (blocks < 1) blocks = 1;
    kern<<<(unsigned)blocks, kBlock, 0, st>>>(b);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

static int epilogue_of(const AggArgs& a) { return a.addend ? kCombine : (a.bias || a.relu) ? kBiasAct : kPlain; }

template <int G, int VPL, int B, int MINB, bool FULL>
static int launch_rows_as(const AggArgs& a, cudaStream_t st) {
    static int bps[3] = {0, 0, 0};
    switch (epilogue_of(a)) {
        case kPlain: return launch_persistent(aggregate_rows_kernel<G, VPL, B, MINB, kPlain, FULL>, &bps[0], a, st);
        case kBiasAct: return launch_persistent(aggregate_rows_kernel<G, VPL, B, MINB, kBiasAct, FULL>, &bps[1], a, st);
        default: return launch_persistent(aggregate_rows_kernel<G, VPL, B, MINB, kCombine, FULL>, &bps[2], a, st);
    }
}
// a narrower 16-byte-aligned width than 4 * G * VPL runs on the same lane layout
template <int G, int VPL, int B, int MINB>
static int launch_rows(const AggArgs& a, cudaStream_t st) {
    return a.f == 4 * G * VPL ? launch_rows_as<G, VPL, B, MINB, true>(a, st) : launch_rows_as<G, VPL, B, MINB, false>(a, st);
}

template <int F>
static int launch_stream(const AggArgs& a, cudaStream_t st) {
    static int bps[3] = {0, 0, 0};
    switch (epilogue_of(a)) {
        case kPlain: return launch_persistent(aggregate_stream_kernel<F, 4, 4, kPlain>, &bps[0], a, st, 4);
        case kBiasAct: return launch_persistent(aggregate_stream_kernel<F, 4, 4, kBiasAct>, &bps[1], a, st, 4);
        default: return launch_persistent(aggregate_stream_kernel<F, 4, 4, kCombine>, &bps[2], a, st, 4);
    }
}

template <int G>
static int launch_narrow(const AggArgs& a, cudaStream_t st) {
    static int bps[2] = {0, 0};
    if (epilogue_of(a) != kPlain) return launch_persistent(aggregate_narrow_kernel<G, true>, &bps[0], a, st);
    return launch_persistent(aggregate_narrow_kernel<G, false>, &bps[1], a, st);
}

// Picks the kernel for a feature width: the vector kernel for the 128-bit-aligned widths it is
// specialised for, the column-strided kernel for everything else.
static int dispatch_aggregate(const AggArgs& a, cudaStream_t st) {
    const int64_t f = a.f;
    const bool vec_ok = (f % 4 == 0) && ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.out) |
                                          reinterpret_cast<uintptr_t>(a.partial) |
                                          reinterpret_cast<uintptr_t>(a.addend)) % 16 == 0);
    // Widths of 32 and 36 to 64 put two or four entries of a row side by side in one warp and add the lane groups'
    // partial sums at the end: that differs from the sequential sum by rounding anyway, so it uses one fused
    // multiply-add per term.  An ordered sum takes the narrow kernel (F <= 32) or the 128-column layout with idle lanes.
    // Row by row or streaming, us (R-MAT unless said):
    //   below eight rows a warp the streaming kernel's start is not paid back: 2.7 k rows, 48 columns, 27 k entries 12.4
    //   against 16.5, 20 k rows, 100 k entries 26 against 30; at 60 k rows it is 56 against 41;
    //   rows of 40 and more entries keep the row kernel's batches full, and out of L2 the streaming kernel is bound by
    //   instructions (40 columns, 170 k rows, 71 entries a row 235 against 278, 38 entries 200 against 175; evenly spread
    //   sources, 300 k rows, 40 entries 220 against 257); with all lanes at work, at 64 columns, the line is at 48 (170 k
    //   rows, 71 entries 257 against 274, 38 entries 211 against 174);
    //   where x does not fit L2 the streaming kernel hides more latency: 64 columns, 2 M rows, 132 M entries 3900
    //   against 3150; at 32 columns it wins for long rows as well (1 M rows, 62 M entries 855 against 780).
    if (vec_ok && !a.ordered && f >= 32 && f <= 64) {
        const bool few = a.n_out < (int64_t)sm_count() * 256;
        const bool lengthy = f > 32 && a.nnz >= a.n_out * (f < 64 ? 40 : 48) && a.n_in * f * 4 <= ((int64_t)(f < 64 ? 100 : 64) << 20);
        if (few || lengthy) return f == 32 ? launch_rows_as<8, 1, 8, 4, true>(a, st) : launch_rows<16, 1, 8, 4>(a, st);
        switch (f) {
            case 32: return launch_stream<32>(a, st);
            case 36: return launch_stream<36>(a, st);
            case 40: return launch_stream<40>(a, st);
            case 44: return launch_stream<44>(a, st);
            case 48: return launch_stream<48>(a, st);
            case 52: return launch_stream<52>(a, st);
            case 56: return launch_stream<56>(a, st);
            case 60: return launch_stream<60>(a, st);
            case 64: return launch_stream<64>(a, st);
        }
    }
    if (vec_ok && f > 32 && f <= 128) return launch_rows<32, 1, 8, 4>(a, st);
    if (vec_ok && f > 128 && f <= 256) return launch_rows<32, 2, 4, 4>(a, st);
    if (vec_ok && f > 256 && f <= 512) return launch_rows<32, 4, 2, 3>(a, st);
    if (f <= 32) {   // narrow rows (any alignment): several rows per warp
        if (f <= 4) return launch_narrow<4>(a, st);
        if (f <= 8) return launch_narrow<8>(a, st);
        if (f <= 16) return launch_narrow<16>(a, st);
        return launch_narrow<32>(a, st);
    }
    static int any2 = 0, any4 = 0, any8 = 0;
    if (f <= 64) return launch_persistent(aggregate_any_kernel<2>, &any2, a, st);
    if (f <= 128) return launch_persistent(aggregate_any_kernel<4>, &any4, a, st);
    return launch_persistent(aggregate_any_kernel<8>, &any8, a, st);
}

}  // namespace jg

using namespace jg;

extern "C" {

size_t jg_spmm_plan_bytes(int64_t n_out, int64_t nnz, int32_t chunk) {
    if (n_out < 0 || nnz < 0 || chunk <= 0) return 0;
    size_t bytes = 0;
    plan_view(nullptr, nnz, chunk, &bytes);
    return bytes;
}

int jg_spmm_plan_build(const int32_t* off, int64_t n_out, int64_t nnz, int32_t chunk, void* plan,
                       size_t plan_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(off && plan, JG_EINVAL, "plan_build: null pointer");
    JG_CHECK_ARG(n_out >= 0 && nnz >= 0 && chunk > 0, JG_EINVAL, "plan_build: bad sizes");
    JG_CHECK_ARG(n_out < INT32_MAX && nnz <= INT32_MAX, JG_ESHAPE, "plan_build: sizes beyond int32");
    size_t need = 0;
    PlanView v = plan_view(plan, nnz, chunk, &need);
    JG_CHECK_ARG(plan_bytes >= need, JG_EWORKSPACE, "plan_build: plan buffer %zu < %zu", plan_bytes, need);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // written by a kernel from its arguments: a copy from this frame would be read at replay under stream capture
    plan_header_kernel<<<1, 1, 0, st>>>(v.hdr, PlanHeader{0, 0, chunk, (int32_t)plan_max_hubs(nnz, chunk),
                                                          (int32_t)plan_max_items(nnz, chunk), {0, 0, 0}});
    JG_LAUNCH_CHECK();
    if (n_out > 0) {
        int grid = (int)((n_out + 255) / 256);
        if (grid > sm_count() * 16) grid = sm_count() * 16;
        plan_build_kernel<<<grid, 256, 0, st>>>(off, n_out, v, chunk);
        JG_LAUNCH_CHECK();
    }
    return JG_OK;
}

size_t jg_aggregate_workspace_bytes(int64_t n_out, int64_t nnz, int64_t f, int32_t chunk) {
    (void)n_out;
    Carver c(nullptr);
    c.take<unsigned long long>(1);
    if (chunk > 0 && nnz > 0 && f > 0) c.take<float>((size_t)plan_max_items(nnz, chunk) * (size_t)f);
    return c.total();
}

static int aggregate_impl(float* out, const float* x, const int32_t* idx, const int32_t* off,
                          const float* w, int64_t n_out, int64_t n_in, int64_t f, int64_t nnz,
                          const void* plan, int32_t chunk, void* workspace, size_t workspace_bytes,
                          jg_stream_t stream, int accumulate, const float* bias = nullptr, int relu = 0, int ordered = 0,
                          int reserve_ctas = 0, const float* addend = nullptr, float scale = 1.f, float add_scale = 0.f) {
    JG_CHECK_ARG(n_out >= 0 && n_in >= 0 && f >= 0 && nnz >= 0, JG_EINVAL, "aggregate: negative size");
    if (n_out == 0 || f == 0) return JG_OK;
    JG_CHECK_ARG(out && off, JG_EINVAL, "aggregate: null out/off");
    JG_CHECK_ARG(nnz == 0 || (x && idx && w), JG_EINVAL, "aggregate: null x/idx/w with nnz > 0");
    JG_CHECK_ARG(n_out < INT32_MAX && n_in <= INT32_MAX && nnz <= kMaxEntries, JG_ESHAPE,
                 "aggregate: sizes beyond int32 indexing");
    JG_CHECK_ARG(!plan || chunk > 0, JG_EINVAL, "aggregate: a plan needs the chunk it was built with");
    JG_CHECK_ARG(workspace, JG_EWORKSPACE, "aggregate: workspace is null");
    const size_t need = jg_aggregate_workspace_bytes(n_out, nnz, f, plan ? chunk : 0);
    JG_CHECK_ARG(workspace_bytes >= need, JG_EWORKSPACE, "aggregate: workspace %zu < %zu", workspace_bytes, need);
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    AggArgs a = {};
    a.out = out; a.x = x; a.idx = idx; a.off = off; a.w = w; a.n_out = n_out; a.f = f;
    a.n_in = n_in; a.nnz = nnz;
    a.accumulate = accumulate;
    a.bias = bias;
    a.relu = relu;
    a.ordered = ordered;
    a.reserve_ctas = reserve_ctas;
    a.addend = addend; a.scale = scale; a.add_scale = add_scale;
    JG_CHECK_ARG(!bias || f % 4 != 0 || reinterpret_cast<uintptr_t>(bias) % 16 == 0, JG_EINVAL,
                 "aggregate: bias must be 16-byte aligned");
    Carver c(workspace);
    a.ticket = c.take<unsigned long long>(1);
    if (plan) {
        PlanView v = plan_view(const_cast<void*>(plan), nnz, chunk, nullptr);
        a.hdr = v.hdr; a.hub_row = v.hub_row; a.hub_first = v.hub_first;
        a.item_hub = v.item_hub; a.item_k = v.item_k;
        a.partial = c.take<float>((size_t)plan_max_items(nnz, chunk) * (size_t)f);
        a.max_items = plan_max_items(nnz, chunk);
    }
    JG_CUDA(cudaMemsetAsync(a.ticket, 0, sizeof(unsigned long long), st));

    int rc = dispatch_aggregate(a, st);
    if (rc != JG_OK) return rc;
    if (plan) {
        hub_fixup_kernel<<<fixup_blocks(nnz, chunk), kBlock, 0, st>>>(a);
        JG_LAUNCH_CHECK();
    }
    return JG_OK;
}


int jg_aggregate_f32(float* out, const float* x, const int32_t* idx, const int32_t* off,
                     const float* w, int64_t n_out, int64_t n_in, int64_t f, int64_t nnz,
                     const void* plan, int32_t chunk, void* workspace, size_t workspace_bytes,
                     jg_stream_t stream) {
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream, 0);
}

int jg_aggregate_add_f32(float* out, const float* x, const int32_t* idx, const int32_t* off,
                         const float* w, int64_t n_out, int64_t n_in, int64_t f, int64_t nnz,
                         const void* plan, int32_t chunk, void* workspace, size_t workspace_bytes,
                         jg_stream_t stream) {
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream, 1);
}

int jg_aggregate_ordered_f32(float* out, const float* x, const int32_t* idx, const int32_t* off, const float* w,
                             int64_t n_out, int64_t n_in, int64_t f, int64_t nnz, const void* plan, int32_t chunk,
                             void* workspace, size_t workspace_bytes, jg_stream_t stream) {
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream, 0, nullptr,
                          0, 1);
}

int jg_aggregate_bias_act_f32(float* out, const float* x, const int32_t* idx, const int32_t* off, const float* w,
                              const float* bias, int relu, int64_t n_out, int64_t n_in, int64_t f, int64_t nnz,
                              const void* plan, int32_t chunk, void* workspace, size_t workspace_bytes, jg_stream_t stream) {
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream, 0, bias,
                          relu ? 1 : 0);
}

int jg_aggregate_combine_f32(float* out, const float* x, const int32_t* idx, const int32_t* off, const float* w,
                             const float* addend, float scale, float add_scale, int64_t n_out, int64_t n_in, int64_t f,
                             int64_t nnz, const void* plan, int32_t chunk, void* workspace, size_t workspace_bytes,
                             jg_stream_t stream) {
    JG_CHECK_ARG(addend || n_out == 0 || f == 0, JG_EINVAL, "aggregate_combine: null addend");
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream, 0, nullptr,
                          0, 0, 0, addend, scale, add_scale);
}

int jg_aggregate_opts_f32(float* out, const float* x, const int32_t* idx, const int32_t* off, const float* w,
                          const float* bias, int relu, int accumulate, int ordered, int reserve_ctas, int64_t n_out,
                          int64_t n_in, int64_t f, int64_t nnz, const void* plan, int32_t chunk, void* workspace,
                          size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(!(accumulate && (bias || relu)), JG_EINVAL, "aggregate_opts: the epilogue cannot be combined with accumulate");
    JG_CHECK_ARG(!(accumulate && ordered), JG_EINVAL, "aggregate_opts: ordered cannot be combined with accumulate");
    JG_CHECK_ARG(reserve_ctas >= 0, JG_EINVAL, "aggregate_opts: negative reserve");
    return aggregate_impl(out, x, idx, off, w, n_out, n_in, f, nnz, plan, chunk, workspace, workspace_bytes, stream,
                          accumulate ? 1 : 0, bias, relu ? 1 : 0, ordered ? 1 : 0, reserve_ctas);
}

// ------------------------------------------------------------------------------------------
// Aggregation without any allocation.
//
// Some callers cannot hand this library a workspace: a host program that is not allowed to call
// cudaMalloc once it is running (an inference server whose memory pool is fixed at start-up, a
// plugin loaded into a process that owns the allocator, code running where a device allocation
// would force a synchronisation it cannot afford).  For them the scratch of the aggregation
// (ticket counter, hub plan, partial rows of split hub rows) lives in one fixed array that is part
// of the library image on every GPU that loads it, kStaticScratchBytes long.
namespace jg {

constexpr size_t kStaticScratchBytes = size_t(32) << 20;  // 32 MiB per GPU, held until exit
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch per device.  In host code the array's name is only a
// stand-in for the symbol, so the address a kernel may use has to be asked for, once per device,
// with that device current.
static unsigned char* g_static_ptr[64] = {nullptr};

static int static_scratch(unsigned char** out) {
    int dev = 0;
    JG_CUDA(cudaGetDevice(&dev));
    JG_CHECK_ARG(dev >= 0 && dev < 64, JG_EUNSUPPORTED, "device index %d beyond 63", dev);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        JG_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        g_static_ptr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_static_ptr[dev];
    return JG_OK;
}

// Start-of-call state of the shared array: ticket at zero, empty plan with this call's piece length.
__global__ void static_scratch_init_kernel(unsigned long long* ticket, PlanHeader* hdr, int32_t chunk, int32_t max_hubs,
                                           int32_t max_items) {
    *ticket = 0ull;
    PlanHeader h = {0, 0, chunk, max_hubs, max_items, {0, 0, 0}};
    *hdr = h;
}

// Bytes of scratch one call needs when hub rows are cut into `chunk`-entry pieces.
static size_t static_need(int64_t nnz, int64_t f, int32_t chunk) {
    size_t plan_bytes = 0;
    plan_view(nullptr, nnz, chunk, &plan_bytes);
    Carver c(nullptr);
    c.take<unsigned long long>(1);
    c.take<unsigned char>(plan_bytes);
    c.take<float>((size_t)plan_max_items(nnz, chunk) * (size_t)f);
    return c.total();
}

}  // namespace jg

size_t jg_aggregate_static_capacity_bytes(void) { return jg::kStaticScratchBytes; }

int jg_aggregate_f32_static(float* out, const float* x, const int32_t* idx, const int32_t* off,
                            const float* w, int64_t n_out, int64_t n_in, int64_t f, int64_t nnz,
                            jg_stream_t stream) {
    JG_CHECK_ARG(n_out >= 0 && n_in >= 0 && f >= 0 && nnz >= 0, JG_EINVAL, "aggregate_static: negative size");
    if (n_out == 0 || f == 0) return JG_OK;
    JG_CHECK_ARG(out && off, JG_EINVAL, "aggregate_static: null out/off");
    JG_CHECK_ARG(nnz == 0 || (x && idx && w), JG_EINVAL, "aggregate_static: null x/idx/w with nnz > 0");
    JG_CHECK_ARG(n_out < INT32_MAX && n_in <= INT32_MAX && nnz <= kMaxEntries, JG_ESHAPE,
                 "aggregate_static: sizes beyond int32 indexing");
    // Piece length: 1024 entries, doubled until plan and partial rows fit the fixed array.
    int32_t chunk = 1024;
    while (static_need(nnz, f, chunk) > kStaticScratchBytes && chunk < (1 << 20)) chunk *= 2;
    const size_t need = static_need(nnz, f, chunk);
    JG_CHECK_ARG(need <= kStaticScratchBytes, JG_EWORKSPACE,
                 "aggregate_static: nnz=%lld at width %lld needs %zu bytes of scratch even with %d-entry pieces; "
                 "the built-in scratch holds %zu (use jg_aggregate_f32 with a caller-owned workspace)",
                 (long long)nnz, (long long)f, need, chunk, kStaticScratchBytes);
    unsigned char* base = nullptr;
    int rc = static_scratch(&base);
    if (rc != JG_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    size_t plan_bytes = 0;
    plan_view(nullptr, nnz, chunk, &plan_bytes);
    Carver c(base);
    AggArgs a = {};
    a.out = out; a.x = x; a.idx = idx; a.off = off; a.w = w; a.n_out = n_out; a.f = f;
    a.n_in = n_in; a.nnz = nnz;
    a.ticket = c.take<unsigned long long>(1);
    PlanView v = plan_view(c.take<unsigned char>(plan_bytes), nnz, chunk, nullptr);
    a.hdr = v.hdr; a.hub_row = v.hub_row; a.hub_first = v.hub_first; a.item_hub = v.item_hub; a.item_k = v.item_k;
    a.partial = c.take<float>((size_t)plan_max_items(nnz, chunk) * (size_t)f);
    a.max_items = plan_max_items(nnz, chunk);

    // The array keeps whatever the previous call left: the two words that must start at zero
    // (ticket, plan counters) are rewritten here; everything else is written before it is read.
    // Both are written by a one-thread kernel from its arguments: no host memory is referenced once
    // this function has returned.
    static_scratch_init_kernel<<<1, 1, 0, st>>>(a.ticket, v.hdr, chunk, (int32_t)plan_max_hubs(nnz, chunk),
                                                (int32_t)plan_max_items(nnz, chunk));
    JG_LAUNCH_CHECK();
    {
        int grid = (int)((n_out + 255) / 256);
        if (grid > sm_count() * 16) grid = sm_count() * 16;
        plan_build_kernel<<<grid, 256, 0, st>>>(off, n_out, v, chunk);
        JG_LAUNCH_CHECK();
    }
    rc = dispatch_aggregate(a, st);
    if (rc != JG_OK) return rc;
    hub_fixup_kernel<<<fixup_blocks(nnz, chunk), kBlock, 0, st>>>(a);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

}  // extern "C"
