// Gradient through a layer's fused epilogue act(y + bias), for sm_100a: the ReLU mask and the bias gradient's
// column sums in one pass over the incoming gradient.
//
//   gm[i,c]  = g[i,c] * (y[i,c] > 0 ? 1 : 0)      (a product, so that a NaN or infinite gradient stays one)
//   gsum[c]  = sum over i of gm[i,c]               (of g itself when there is no mask)
//
// Stands for the elementwise passes and the reduction that the reference's autograd runs after its layers
// (nn/conv/gcn_conv.py:96-101, examples/gcn_example.py:76).  HBM-bound: g and y are read once, gm written once;
// compare, multiply and column sum as separate passes moved the same rows seven times.
// A block takes consecutive rows; a thread owns V = 4 or 1 neighbouring columns and every TY-th row, four rows in
// flight, in four accumulators.  Blocks' sums are added in a fixed order by the slice reduction: no atomics,
// identical results run to run.
// 170 k x 256: 0.29 ms (compare, multiply, column sum) before, 0.13 ms here.
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

// tx: threads along the columns (a power of two), 256 / tx rows side by side.
template <int V>
__global__ void __launch_bounds__(kReluThreads) relu_grad_kernel(float* __restrict__ gm, float* __restrict__ partial,
                                                                 const float* __restrict__ g, const float* __restrict__ y, int64_t n,
                                                                 int64_t f, int tx, int64_t rows_per_block) {
    constexpr int U = 4;
    __shared__ Cols<V> s_sum[kReluThreads];
    const int ty = kReluThreads / tx, c = threadIdx.x % tx, r = threadIdx.x / tx;
    const int64_t vecs = f / V;
    const int64_t r0 = (int64_t)blockIdx.x * rows_per_block;
    const int64_t r1 = r0 + rows_per_block < n ? r0 + rows_per_block : n;
    for (int64_t cb = 0; cb < vecs; cb += tx) {
        const int64_t cv = cb + c;
        Cols<V> acc[U];
#pragma unroll
        for (int u = 0; u < U; u++) acc[u].zero();
        if (cv < vecs) {
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
                    if (y) a[u].mask(b[u]);
                    if (gm) a[u].store(gm + i * f + cv * V);
                    acc[u].add(a[u]);
                }
            }
        }
        if (partial) {
            acc[0].add(acc[1]);
            acc[2].add(acc[3]);
            acc[0].add(acc[2]);
            s_sum[threadIdx.x] = acc[0];
            __syncthreads();
            if (r == 0 && cv < vecs) {
                for (int k = 1; k < ty; k++) acc[0].add(s_sum[k * tx + c]);
                acc[0].store(partial + (int64_t)blockIdx.x * f + cv * V);
            }
            __syncthreads();
        }
    }
}

// Blocks (and partial sums): four per SM, but at least 32 rows each, so that a small batch does not pay for sums of sums.
static int64_t relu_blocks(int64_t n) {
    int64_t b = (n + 31) / 32;
    const int64_t most = (int64_t)sm_count() * 4;
    return b > most ? most : (b < 1 ? 1 : b);
}

}  // namespace jg

using namespace jg;

extern "C" {

size_t jg_relu_grad_workspace_bytes(int64_t n, int64_t f) {
    if (n <= 0 || f <= 0) return 0;
    return align_up((size_t)relu_blocks(n) * (size_t)f * sizeof(float), 256);
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
    const int64_t blocks = relu_blocks(n);
    const int64_t rows = (n + blocks - 1) / blocks;
    float* partial = gsum ? static_cast<float*>(workspace) : nullptr;
    const uintptr_t all = reinterpret_cast<uintptr_t>(gm) | reinterpret_cast<uintptr_t>(partial) | reinterpret_cast<uintptr_t>(g) |
                          reinterpret_cast<uintptr_t>(y);
    const bool vec = f % 4 == 0 && all % 16 == 0;
    const int64_t vecs = vec ? f / 4 : f;
    int tx = 1;
    while (tx < kReluThreads && tx < vecs) tx *= 2;
    if (vec) relu_grad_kernel<4><<<(unsigned)blocks, kReluThreads, 0, st>>>(gm, partial, g, y, n, f, tx, rows);
    else relu_grad_kernel<1><<<(unsigned)blocks, kReluThreads, 0, st>>>(gm, partial, g, y, n, f, tx, rows);
    JG_LAUNCH_CHECK();
    return gsum ? reduce_slices(gsum, partial, 1, f, (int)blocks, st) : JG_OK;
}

}  // extern "C"
