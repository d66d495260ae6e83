// Gradient through a layer's fused epilogue act(y + bias), for sm_100a: the ReLU mask and the bias gradient's
// column sums in one pass over the incoming gradient.
//
//   gm[i,c]  = g[i,c] * (y[i,c] > 0 ? 1 : 0)      (a product, so that a NaN or infinite gradient stays one)
//   gsum[c]  = sum over i of gm[i,c]               (of g itself when there is no mask)
//
// Stands for the elementwise passes and the reduction that the reference's autograd runs after its layers
// (nn/conv/gcn_conv.py:96-101, examples/gcn_example.py:76).  HBM-bound: g and y are read once, gm written once;
// compare, multiply and column sum as separate passes moved the same rows seven times.
// Without the sums the rows do not matter: the arrays are one run of values, 16 bytes a lane at any width.  With them a
// block takes consecutive rows and a slab of lanes' columns; a lane owns V = 4, 2 or 1 neighbouring columns
// (what the width and the bases are aligned to) and every ty-th row, U of them in flight, each in an accumulator.
// Blocks' sums are added in a fixed order by the slice reduction (a short input is one block, which stores them):
// no atomics, identical results run to run.
// 170 k x 256, compare + multiply + column sum against this: 0.293 / 0.126 ms, without the sum 0.170 / 0.082; 170 k x 130
// 0.142 / 0.118 and 0.089 / 0.042; 64 x 4096 9.5 / 4.9 and 5.5 / 2.1 us; 2708 x 7 9.5 / 5.3 us.
#include "common.cuh"

namespace jg {

int reduce_slices(float* c, const float* partial, int64_t M, int64_t N, int slices, cudaStream_t st);

constexpr int kReluThreads = 256;

template <int V> struct Cols;
template <> struct Cols<1> {
    float x;
    __device__ __forceinline__ void load(const float* p) { x = __ldg(p); }
    __device__ __forceinline__ void store(float* p) const { *p = x; }
    __device__ __forceinline__ void zero() { x = 0.f; }
    __device__ __forceinline__ void mask(const Cols& y) { x *= y.x > 0.f ? 1.f : 0.f; }
    __device__ __forceinline__ void add(const Cols& o) { x += o.x; }
};
template <> struct Cols<2> {
    float2 x;
    __device__ __forceinline__ void load(const float* p) { x = __ldg(reinterpret_cast<const float2*>(p)); }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float2*>(p) = x; }
    __device__ __forceinline__ void zero() { x = make_float2(0.f, 0.f); }
    __device__ __forceinline__ void mask(const Cols& y) { x.x *= y.x.x > 0.f ? 1.f : 0.f; x.y *= y.x.y > 0.f ? 1.f : 0.f; }
    __device__ __forceinline__ void add(const Cols& o) { x.x += o.x.x; x.y += o.x.y; }
};
template <> struct Cols<4> {
    float4 x;
    __device__ __forceinline__ void load(const float* p) { x = __ldg(reinterpret_cast<const float4*>(p)); }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = x; }
    __device__ __forceinline__ void zero() { x = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void mask(const Cols& y) {
        x.x *= y.x.x > 0.f ? 1.f : 0.f; x.y *= y.x.y > 0.f ? 1.f : 0.f;
        x.z *= y.x.z > 0.f ? 1.f : 0.f; x.w *= y.x.w > 0.f ? 1.f : 0.f;
    }
    __device__ __forceinline__ void add(const Cols& o) { x.x += o.x.x; x.y += o.x.y; x.z += o.x.z; x.w += o.x.w; }
};

// The mask alone: `count` values as groups of V (4 where the bases allow, else 1) and a tail of single ones.
template <int V>
__global__ void __launch_bounds__(kReluThreads) relu_mask_kernel(float* __restrict__ gm, const float* __restrict__ g,
                                                                 const float* __restrict__ y, int64_t count) {
    constexpr int U = 2;
    const int64_t step = (int64_t)gridDim.x * kReluThreads, me = (int64_t)blockIdx.x * kReluThreads + threadIdx.x;
    const int64_t groups = count / V;
    for (int64_t i0 = me; i0 < groups; i0 += U * step) {
        Cols<V> a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t i = i0 + u * step;
            if (i < groups) { a[u].load(g + i * V); b[u].load(y + i * V); }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t i = i0 + u * step;
            if (i < groups) { a[u].mask(b[u]); a[u].store(gm + i * V); }
        }
    }
    if (me < count - groups * V) {
        const int64_t i = groups * V + me;
        gm[i] = __ldg(g + i) * (__ldg(y + i) > 0.f ? 1.f : 0.f);
    }
}

// Mask and column sums.  A slab of tx lanes along the columns, T / tx rows side by side; blockIdx.x: slab,
// blockIdx.y: rows.  `sums`: [gridDim.y, f].
template <int V>
constexpr int kRowsInFlight = V == 4 ? 4 : 8;
template <int V, int T>
__global__ void __launch_bounds__(T) relu_grad_kernel(float* __restrict__ gm, float* __restrict__ sums, const float* __restrict__ g,
                                                      const float* __restrict__ y, int64_t n, int64_t f, int tx,
                                                      int64_t rows_per_block) {
    constexpr int U = kRowsInFlight<V>;
    __shared__ Cols<V> s_sum[T];
    const int ty = T / tx, c = threadIdx.x % tx, r = threadIdx.x / tx;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_block;
    const int64_t r1 = r0 + rows_per_block < n ? r0 + rows_per_block : n;
    const int64_t cv = (int64_t)blockIdx.x * tx + c;
    const bool mine = r < ty && cv < f / V;
    Cols<V> acc[U];
#pragma unroll
    for (int u = 0; u < U; u++) acc[u].zero();
    if (mine) {
        for (int64_t row = r0 + r; row < r1; row += (int64_t)U * ty) {
            Cols<V> a[U], b[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int64_t i = row + (int64_t)u * ty;
                a[u].zero();
                b[u].zero();
                if (i < r1) {
                    a[u].load(g + i * f + cv * V);
                    if (y) b[u].load(y + i * f + cv * V);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int64_t i = row + (int64_t)u * ty;
                if (i >= r1) continue;
                if (y) {
                    a[u].mask(b[u]);
                    if (gm) a[u].store(gm + i * f + cv * V);
                }
                acc[u].add(a[u]);
            }
        }
    }
#pragma unroll
    for (int o = U / 2; o > 0; o /= 2)
#pragma unroll
        for (int u = 0; u < o; u++) acc[u].add(acc[u + o]);
    s_sum[threadIdx.x] = acc[0];
    int half = 1;
    while (half < ty) half *= 2;
    for (half /= 2; half > 0; half /= 2) {     // rows r and r + half, in the same order whatever the block
        __syncthreads();
        if (r < half && r + half < ty) s_sum[threadIdx.x].add(s_sum[(r + half) * tx + c]);
    }
    if (mine && r == 0) s_sum[c].store(sums + (int64_t)blockIdx.y * f + cv * V);
}

// How a call with sums is split into slabs of columns and blocks of rows.
constexpr int kFewThreads = 256, kManyThreads = 512;
struct ReluSplit {
    bool many;
    int tx;
    int64_t slabs, blocks;
};
template <int V>
static ReluSplit relu_split(int64_t n, int64_t f) {
    ReluSplit s;
    // wide slabs read long stretches of a row (60 k x 602: 248 us with slabs of 31 lanes), narrow ones occupy more SMs
    s.many = n >= 8192;
    const int threads = s.many ? kManyThreads : kFewThreads, widest = s.many ? threads / 2 : 32;
    const int64_t vecs = f / V;
    s.slabs = (vecs + widest - 1) / widest;
    s.tx = (int)((vecs + s.slabs - 1) / s.slabs);
    // 1024 threads per SM over all slabs, each at least one batch of rows (so a short input is one block)
    const int64_t least = (int64_t)(threads / s.tx) * kRowsInFlight<V>;
    const int64_t want = (n + least - 1) / least, most = ((int64_t)sm_count() * (1024 / threads) + s.slabs - 1) / s.slabs;
    s.blocks = want < most ? want : most;
    return s;
}
template <int V>
static int launch_relu(float* gm, float* gsum, float* partial, const float* g, const float* y, int64_t n, int64_t f, cudaStream_t st) {
    const ReluSplit s = relu_split<V>(n, f);
    const dim3 grid((unsigned)s.slabs, (unsigned)s.blocks);
    float* sums = s.blocks == 1 ? gsum : partial;
    const int64_t rows = (n + s.blocks - 1) / s.blocks;
    if (s.many) relu_grad_kernel<V, kManyThreads><<<grid, kManyThreads, 0, st>>>(gm, sums, g, y, n, f, s.tx, rows);
    else relu_grad_kernel<V, kFewThreads><<<grid, kFewThreads, 0, st>>>(gm, sums, g, y, n, f, s.tx, rows);
    JG_LAUNCH_CHECK();
    return s.blocks == 1 ? JG_OK : reduce_slices(gsum, partial, 1, f, (int)s.blocks, st);
}

}  // namespace jg

using namespace jg;

extern "C" {

size_t jg_relu_grad_workspace_bytes(int64_t n, int64_t f) {
    if (n <= 0 || f <= 0) return 0;
    // the widest access that f allows depends on the bases too: room for whichever is taken
    int64_t blocks = relu_split<1>(n, f).blocks;
    if (f % 2 == 0 && relu_split<2>(n, f).blocks > blocks) blocks = relu_split<2>(n, f).blocks;
    if (f % 4 == 0 && relu_split<4>(n, f).blocks > blocks) blocks = relu_split<4>(n, f).blocks;
    return align_up((size_t)blocks * (size_t)f * sizeof(float), 256);
}

int jg_relu_grad_f32(float* gm, float* gsum, const float* g, const float* y, int64_t n, int64_t f, void* workspace,
                     size_t workspace_bytes, jg_stream_t stream) {
    JG_CHECK_ARG(n >= 0 && f >= 0, JG_EINVAL, "relu_grad: negative size");
    JG_CHECK_ARG(!gm || y || n == 0, JG_EINVAL, "relu_grad: a masked gradient needs the layer's output");
    if (f == 0 || (!gm && !gsum)) return JG_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n == 0) {
        if (gsum) JG_CUDA(cudaMemsetAsync(gsum, 0, (size_t)f * sizeof(float), st));
        return JG_OK;
    }
    JG_CHECK_ARG(g, JG_EINVAL, "relu_grad: null gradient");
    JG_CHECK_ARG(f < ((int64_t)1 << 31) && n < ((int64_t)1 << 40), JG_ESHAPE, "relu_grad: size out of range");
    JG_CHECK_ARG(!gsum || (workspace && workspace_bytes >= jg_relu_grad_workspace_bytes(n, f)), JG_EWORKSPACE,
                 "relu_grad: workspace %zu < %zu", workspace_bytes, jg_relu_grad_workspace_bytes(n, f));
    const uintptr_t data = reinterpret_cast<uintptr_t>(gm) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(y);
    if (!gsum) {
        const int64_t count = n * f, per = (data % 16 == 0 ? 4 : 1) * 2 * (int64_t)kReluThreads;
        int64_t blocks = (count + per - 1) / per;
        if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
        if (data % 16 == 0) relu_mask_kernel<4><<<(unsigned)blocks, kReluThreads, 0, st>>>(gm, g, y, count);
        else relu_mask_kernel<1><<<(unsigned)blocks, kReluThreads, 0, st>>>(gm, g, y, count);
        JG_LAUNCH_CHECK();
        return JG_OK;
    }
    float* partial = static_cast<float*>(workspace);
    const uintptr_t all = data | reinterpret_cast<uintptr_t>(partial) | reinterpret_cast<uintptr_t>(gsum);
    if (f % 4 == 0 && all % 16 == 0) return launch_relu<4>(gm, gsum, partial, g, y, n, f, st);
    if (f % 2 == 0 && all % 8 == 0) return launch_relu<2>(gm, gsum, partial, g, y, n, f, st);
    return launch_relu<1>(gm, gsum, partial, g, y, n, f, st);
}

}  // extern "C"
