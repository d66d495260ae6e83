// Dense products in full fp32 on the CUDA cores (sm_100a): C[M,N] = op(A) * op(B) (+ bias, ReLU).
//
// The reference's layers hand `x @ self.weight` and its two gradient products to the runtime, which
// calls cuBLAS (nn/conv/gcn_conv.py:95, nn/conv/gat_conv.py:86).  The tensor-core kernel
// (gemm.cu, TF32 products) is the transform of the hot path; this kernel serves what it does not:
// the fp32 opt-out of the layers (comparisons at 1e-5 need fp32 products), the weight gradient
// x^T * g (a reduction over the rows, the one operand layout the row-tiled kernel does not take) and
// shapes the tensor-core kernel refuses.  With it no product of the path goes to a library.
//
// Operands are addressed by two strides each, A(i,l) = a[i*sa0 + l*sa1], B(l,j) = b[l*sb0 + j*sb1].
// sgemm_kernel takes any strides (x @ W, g @ W^T): 64x64 output tile per CTA, 16-deep slices through shared
// memory, 4x4 register block per thread, fp32 FMA.  sgemm_tn_kernel takes x^T @ g, both operands along their
// rows.  A long reduction (millions of rows) is cut into slices across CTAs whose partial tiles are added in a
// fixed order by a second kernel: no atomics, identical results run to run.
#include "common.cuh"

namespace jg {

constexpr int kBM = 64, kBN = 64, kBK = 16;

struct SgemmArgs {
    float* c;             // output [M, ldc] (single slice) or partial tiles [slices][M][N]
    const float* a;
    const float* b;
    const float* bias;    // [N] or null (single slice only; else applied by the reduction)
    int64_t M, N, K;
    int64_t sa0, sa1, sb0, sb1, ldc;
    int64_t k_slice;      // reduction length per slice (a multiple of kBK)
    int relu;
    int slices;
};

__global__ void __launch_bounds__(256) sgemm_kernel(SgemmArgs g) {
    __shared__ float As[kBK][kBM + 4];
    __shared__ float Bs[kBK][kBN + 4];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int64_t i0 = (int64_t)blockIdx.x * kBM, j0 = (int64_t)blockIdx.y * kBN;
    const int64_t l_begin = (int64_t)blockIdx.z * g.k_slice;
    const int64_t l_end = l_begin + g.k_slice < g.K ? l_begin + g.k_slice : g.K;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[r][c] = 0.f;
    const bool a_rows_contig = g.sa0 == 1;     // consecutive i adjacent in memory (A given transposed)
    const bool b_cols_contig = g.sb1 == 1;     // consecutive j adjacent in memory
    for (int64_t l0 = l_begin; l0 < l_end; l0 += kBK) {
#pragma unroll
        for (int e = tid; e < kBM * kBK; e += 256) {
            const int ii = a_rows_contig ? e % kBM : e / kBK;
            const int ll = a_rows_contig ? e / kBM : e % kBK;
            const int64_t i = i0 + ii, l = l0 + ll;
            As[ll][ii] = (i < g.M && l < l_end) ? __ldg(g.a + i * g.sa0 + l * g.sa1) : 0.f;
        }
#pragma unroll
        for (int e = tid; e < kBN * kBK; e += 256) {
            const int jj = b_cols_contig ? e % kBN : e / kBK;
            const int ll = b_cols_contig ? e / kBN : e % kBK;
            const int64_t j = j0 + jj, l = l0 + ll;
            Bs[ll][jj] = (j < g.N && l < l_end) ? __ldg(g.b + l * g.sb0 + j * g.sb1) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int l = 0; l < kBK; l++) {
            const float4 av = *reinterpret_cast<const float4*>(&As[l][ty * 4]);
            const float4 bv = *reinterpret_cast<const float4*>(&Bs[l][tx * 4]);
            const float a4[4] = {av.x, av.y, av.z, av.w}, b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[r][c] = fmaf(a4[r], b4[c], acc[r][c]);
        }
        __syncthreads();
    }
    const bool single = g.slices == 1;
    float* out = single ? g.c : g.c + (size_t)blockIdx.z * (size_t)g.M * (size_t)g.N;
    const int64_t ld = single ? g.ldc : g.N;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int64_t i = i0 + ty * 4 + r;
        if (i >= g.M) continue;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int64_t j = j0 + tx * 4 + c;
            if (j >= g.N) continue;
            float v = acc[r][c];
            if (single) {
                if (g.bias) v += __ldg(g.bias + j);
                if (g.relu) v = fmaxf(v, 0.f);
            }
            out[i * ld + j] = v;
        }
    }
}

// ---- x^T * g: both operands read along their rows ------------------------------------------------------------
// C[i, j] = sum over rows l of a[l, i] * b[l, j], a [K, M] and b [K, N] with unit column strides: the weight gradient
// at widths the tensor-core kernel does not take (TMA cannot address rows of 602, 1433 or 47 floats), and of the
// fp32 layers.  Bound by the fp32 FMA rate: 128 x 16 TN outputs per CTA, 8 x TN per thread, products as packed
// pairs (two FMAs per instruction), rows of both operands copied into a three-stage shared-memory ring as they
// are (cp.async of 4 to 16 bytes, as far as the row pitch is aligned), so nothing is transposed.  One wave of CTAs:
// the slices of the row range fill the device twice over and are added by sgemm_reduce_kernel.
// Against the 64 x 64 kernel above: 233 k rows, 602 x 64 columns 1.41 -> 0.38 ms (47 TFLOP/s); 170 k rows, 256 x 47
// 0.39 -> 0.115 ms; 2708 rows, 1433 x 256 0.115 -> 0.06 ms.
constexpr int kTnM = 128, kTnK = 16, kTnStages = 3;

__device__ __forceinline__ void cp_async_bytes(void* dst, const float* src, int bytes, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = in ? bytes : 0;      // the rest of the destination is zero-filled
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else if (bytes == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// AV, BV: floats per copy of a row of a and of b (4, 2, 1: pitch and base are multiples of that many).
template <int TN, int AV, int BV>
__global__ void __launch_bounds__(256, 2) sgemm_tn_kernel(SgemmArgs g) {
    constexpr int BN = 16 * TN;
    extern __shared__ __align__(16) float tn_smem[];
    float* As = tn_smem;                                  // [stages][kTnK][kTnM]
    float* Bs = tn_smem + kTnStages * kTnK * kTnM;        // [stages][kTnK][BN]
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int64_t i0 = (int64_t)blockIdx.x * kTnM, j0 = (int64_t)blockIdx.y * BN;
    const int64_t l_begin = (int64_t)blockIdx.z * g.k_slice;
    const int64_t l_end = l_begin + g.k_slice < g.K ? l_begin + g.k_slice : g.K;
    const int steps = l_end > l_begin ? (int)((l_end - l_begin + kTnK - 1) / kTnK) : 0;

    auto fill = [&](int step) {
        float* as = As + (step % kTnStages) * kTnK * kTnM;
        float* bs = Bs + (step % kTnStages) * kTnK * BN;
        const int64_t l0 = l_begin + (int64_t)step * kTnK;
        constexpr int AR = kTnM / AV, BR = BN / BV;       // copies per row
#pragma unroll
        for (int e = tid; e < kTnK * AR; e += 256) {
            const int ll = e / AR, ii = (e % AR) * AV;
            const bool in = l0 + ll < l_end && i0 + ii < g.M;
            cp_async_bytes(as + ll * kTnM + ii, in ? g.a + (l0 + ll) * g.sa1 + i0 + ii : g.a, 4 * AV, in);
        }
#pragma unroll
        for (int e = tid; e < kTnK * BR; e += 256) {
            const int ll = e / BR, jj = (e % BR) * BV;
            const bool in = l0 + ll < l_end && j0 + jj < g.N;
            cp_async_bytes(bs + ll * BN + jj, in ? g.b + (l0 + ll) * g.sb0 + j0 + jj : g.b, 4 * BV, in);
        }
    };

    unsigned long long acc[4][TN];                        // rows ty*8 + 2r and 2r + 1, column tx + 16 c or tx * TN + c
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < TN; c++) acc[r][c] = 0ull;
#pragma unroll
    for (int s = 0; s < kTnStages - 1; s++) {
        if (s < steps) fill(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int step = 0; step < steps; step++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kTnStages - 2) : "memory");
        __syncthreads();                                  // this stage has landed, and nobody reads the one filled next
        if (step + kTnStages - 1 < steps) fill(step + kTnStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = As + (step % kTnStages) * kTnK * kTnM + ty * 8;
        const float* bs = Bs + (step % kTnStages) * kTnK * BN;
#pragma unroll
        for (int l = 0; l < kTnK; l++) {
            const ulonglong2 a01 = *reinterpret_cast<const ulonglong2*>(as + l * kTnM);
            const ulonglong2 a23 = *reinterpret_cast<const ulonglong2*>(as + l * kTnM + 4);
            const unsigned long long a[4] = {a01.x, a01.y, a23.x, a23.y};
            float b[TN];
            if constexpr (TN % 4 == 0) {
#pragma unroll
                for (int c = 0; c < TN; c += 4) {         // columns 4 tx .. of each 64-column half: a quarter-warp reads 128 bytes
                    const float4 v = *reinterpret_cast<const float4*>(bs + l * BN + (c / 4) * 64 + tx * 4);
                    b[c] = v.x; b[c + 1] = v.y; b[c + 2] = v.z; b[c + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < TN; c++) b[c] = bs[l * BN + c * 16 + tx];
            }
#pragma unroll
            for (int c = 0; c < TN; c++) {
                const unsigned long long bb = pack2(b[c], b[c]);
#pragma unroll
                for (int r = 0; r < 4; r++) fma2(acc[r][c], a[r], bb);
            }
        }
    }
    const bool single = g.slices == 1;
    float* out = single ? g.c : g.c + (size_t)blockIdx.z * (size_t)g.M * (size_t)g.N;
    const int64_t ld = single ? g.ldc : g.N;
    const bool vec = g.N % 4 == 0 && ld % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
    auto finish = [&](int r, int c, int64_t j) {
        const unsigned long long p = acc[r / 2][c];
        float v = __uint_as_float((unsigned)(r % 2 ? p >> 32 : p));
        if (single) {
            if (g.bias) v += __ldg(g.bias + j);
            if (g.relu) v = fmaxf(v, 0.f);
        }
        return v;
    };
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int64_t i = i0 + ty * 8 + r;
        if (i >= g.M) continue;
        if constexpr (TN % 4 == 0) {
            if (vec) {       // four columns of a thread lie side by side
#pragma unroll
                for (int c = 0; c < TN; c += 4) {
                    const int64_t j = j0 + (c / 4) * 64 + tx * 4;
                    if (j < g.N) *reinterpret_cast<float4*>(out + i * ld + j) =
                        make_float4(finish(r, c, j), finish(r, c + 1, j + 1), finish(r, c + 2, j + 2), finish(r, c + 3, j + 3));
                }
                continue;
            }
        }
#pragma unroll
        for (int c = 0; c < TN; c++) {
            const int64_t j = j0 + (TN % 4 == 0 ? (c / 4) * 64 + tx * 4 + c % 4 : c * 16 + tx);
            if (j >= g.N) continue;
            out[i * ld + j] = finish(r, c, j);
        }
    }
}

// Columns per CTA (16 TN): the padded width, weighed with how well the inner loop of that TN feeds the FMAs
// (shared-memory reads per product).
static int tn_cols(int64_t N) {
    const int tn[5] = {1, 2, 3, 4, 8};
    const double rate[5] = {0.45, 0.65, 0.8, 0.9, 1.0};
    int best = 8;
    double cost = 1e300;
    for (int k = 0; k < 5; k++) {
        const int64_t bn = 16 * tn[k];
        const double c = (double)((N + bn - 1) / bn * bn) / rate[k];
        if (c <= cost) { cost = c; best = tn[k]; }
    }
    return best;
}
static int tn_row_slices(int64_t M, int64_t N, int64_t K) {
    const int64_t bn = 16 * tn_cols(N);
    const int64_t tiles = ((M + kTnM - 1) / kTnM) * ((N + bn - 1) / bn);
    int64_t want = 2 * (int64_t)sm_count() / tiles;                      // one wave of two CTAs per SM
    const int64_t most = (K + 4 * kTnK - 1) / (4 * kTnK);                // at least four steps each
    if (want > most) want = most;
    return want < 1 ? 1 : (int)want;
}

// A few CTAs of 128 x 128 outputs each take longer than the many 64 x 64 tiles of the kernel above: 16 rows, 1433 x 256
// columns 6.2 us against 4.0, 1000 rows, 47 x 256 12.6 against 11.0.  From a quarter of the SMs on, and with narrower
// tiles at any count, it is the faster one (128 rows, 1433 x 256, 48 CTAs: 14.6 both; 500 rows, 64 x 64, 8 CTAs: 8.8 against 10.9).
static bool tn_pays(int64_t M, int64_t N, int64_t K) {
    const int cols = tn_cols(N);
    const int64_t tiles = ((M + kTnM - 1) / kTnM) * ((N + 16 * cols - 1) / (16 * cols));
    return cols < 8 || tiles * tn_row_slices(M, N, K) * 4 >= sm_count();
}

static int copy_floats(const float* p, int64_t pitch) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(p);
    return pitch % 4 == 0 && b % 16 == 0 ? 4 : (pitch % 2 == 0 && b % 8 == 0 ? 2 : 1);
}

template <int TN, int AV>
static void launch_tn_b(const SgemmArgs& g, int bv, dim3 grid, size_t smem, cudaStream_t st) {
    // a copy never crosses the row's end: width and pitch are the same number here
    if (TN % 4 == 0 && bv == 4) sgemm_tn_kernel<TN, AV, 4><<<grid, 256, smem, st>>>(g);
    else sgemm_tn_kernel<TN, AV, 1><<<grid, 256, smem, st>>>(g);
}
template <int TN>
static void launch_tn(const SgemmArgs& g, cudaStream_t st) {
    const dim3 grid((unsigned)((g.M + kTnM - 1) / kTnM), (unsigned)((g.N + 16 * TN - 1) / (16 * TN)), (unsigned)g.slices);
    const size_t smem = (size_t)kTnStages * kTnK * (kTnM + 16 * TN) * sizeof(float);
    const int av = g.M % 4 == 0 ? copy_floats(g.a, g.sa1) : (g.M % 2 == 0 && copy_floats(g.a, g.sa1) >= 2 ? 2 : 1);
    const int bv = g.N % 4 == 0 ? copy_floats(g.b, g.sb0) : 1;
    if (av == 4) launch_tn_b<TN, 4>(g, bv, grid, smem, st);
    else if (av == 2) launch_tn_b<TN, 2>(g, bv, grid, smem, st);
    else launch_tn_b<TN, 1>(g, bv, grid, smem, st);
}

// C = sum of the slices' partial tiles in slice order (+ bias, ReLU), one thread per output.
__global__ void __launch_bounds__(256) sgemm_reduce_few_kernel(float* __restrict__ c, const float* __restrict__ partial, int64_t M,
                                                               int64_t N, int64_t ldc, int slices, const float* __restrict__ bias,
                                                               int relu) {
    const size_t mn = (size_t)(M * N);
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < M * N; t += (int64_t)gridDim.x * blockDim.x) {
        float v = __ldg(partial + t);
#pragma unroll 8
        for (int s = 1; s < slices; s++) v = __fadd_rn(v, __ldg(partial + (size_t)s * mn + t));
        const int64_t i = t / N, j = t - i * N;
        if (bias) v += __ldg(bias + j);
        if (relu) v = fmaxf(v, 0.f);
        c[i * ldc + j] = v;
    }
}

// The same for many slices of few outputs.  32 outputs per block; eight groups of threads add an eighth of the slices each, in order, and the eighths are
// added in order: with one thread per output, 148 slices of a 128 x 128 gradient were a chain of 148 loads.
__global__ void __launch_bounds__(256) sgemm_reduce_kernel(float* __restrict__ c, const float* __restrict__ partial, int64_t M,
                                                           int64_t N, int64_t ldc, int slices, const float* __restrict__ bias, int relu) {
    constexpr int kGroups = 8;
    __shared__ float s_sum[kGroups][32];
    const int lane = threadIdx.x % 32, grp = threadIdx.x / 32;
    const int per = (slices + kGroups - 1) / kGroups;
    const int s0 = grp * per, s1 = s0 + per < slices ? s0 + per : slices;
    const size_t mn = (size_t)(M * N);
    for (int64_t t0 = (int64_t)blockIdx.x * 32; t0 < M * N; t0 += (int64_t)gridDim.x * 32) {
        const int64_t t = t0 + lane;
        float v = 0.f;
        if (t < M * N) {
#pragma unroll 8
            for (int s = s0; s < s1; s++) v = __fadd_rn(v, __ldg(partial + (size_t)s * mn + t));
        }
        s_sum[grp][lane] = v;
        __syncthreads();
        if (grp == 0 && t < M * N) {
#pragma unroll
            for (int q = 1; q < kGroups; q++) v = __fadd_rn(v, s_sum[q][lane]);
            const int64_t i = t / N, j = t - i * N;
            if (bias) v += __ldg(bias + j);
            if (relu) v = fmaxf(v, 0.f);
            c[i * ldc + j] = v;
        }
        __syncthreads();
    }
}

// The second kernel's barriers cost more than the chain they cut where the first fills the device by itself: from 2^17
// outputs on, or from 2^15 with two loads or less in each of the groups (2708 x 256 outputs, two slices: 5 us against 15;
// 1432 x 256, three: 4 against 11; 64 x 64, eight: 3 against 2).
static int launch_reduce(float* c, const float* partial, int64_t M, int64_t N, int64_t ldc, int slices, const float* bias, int relu,
                         cudaStream_t st) {
    const bool few = M * N >= (int64_t)1 << 17 || (M * N > (int64_t)1 << 15 && slices <= 16);
    const int64_t per_block = few ? 256 : 32;
    int64_t blocks = (M * N + per_block - 1) / per_block;
    if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
    if (few) sgemm_reduce_few_kernel<<<(unsigned)blocks, 256, 0, st>>>(c, partial, M, N, ldc, slices, bias, relu);
    else sgemm_reduce_kernel<<<(unsigned)blocks, 256, 0, st>>>(c, partial, M, N, ldc, slices, bias, relu);
    JG_LAUNCH_CHECK();
    return JG_OK;
}

// Used by the tensor-core weight gradient as well: c[M, N] = sum of `slices` partial results, in order.
int reduce_slices(float* c, const float* partial, int64_t M, int64_t N, int slices, cudaStream_t st) {
    return launch_reduce(c, partial, M, N, N, slices, nullptr, 0, st);
}

static int sgemm_slices(int64_t M, int64_t N, int64_t K) {
    const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN);
    int64_t want = (2 * (int64_t)sm_count() + tiles - 1) / tiles;      // enough CTAs to fill the device twice
    const int64_t most = (K + 4 * kBK - 1) / (4 * kBK);                  // at least four slices' worth of work each
    if (want > most) want = most;
    if (want > 1024) want = 1024;
    return want < 1 ? 1 : (int)want;
}

}  // namespace jg

using namespace jg;

extern "C" {

size_t jg_gemm_f32_workspace_bytes(int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int s1 = sgemm_slices(M, N, K), s2 = tn_row_slices(M, N, K);
    const int s = s1 > s2 ? s1 : s2;       // whichever kernel the strides select
    return s > 1 ? align_up((size_t)s * (size_t)M * (size_t)N * sizeof(float), 256) : 0;
}

int jg_gemm_f32(float* c, const float* a, const float* b, const float* bias, int64_t M, int64_t N, int64_t K, int64_t sa0,
                int64_t sa1, int64_t sb0, int64_t sb1, int64_t ldc, int relu, void* workspace, size_t workspace_bytes,
                jg_stream_t stream) {
    JG_CHECK_ARG(M >= 0 && N >= 0 && K >= 0 && ldc >= N, JG_EINVAL, "gemm_f32: bad size");
    if (M == 0 || N == 0) return JG_OK;
    JG_CHECK_ARG(c && (K == 0 || (a && b)), JG_EINVAL, "gemm_f32: null pointer");
    JG_CHECK_ARG((N + kBN - 1) / kBN < 65536 && (M + kBM - 1) / kBM < 2147483647, JG_ESHAPE, "gemm_f32: output too large");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    SgemmArgs g = {};
    g.a = a; g.b = b; g.bias = bias; g.M = M; g.N = N; g.K = K;
    g.sa0 = sa0; g.sa1 = sa1; g.sb0 = sb0; g.sb1 = sb1; g.ldc = ldc; g.relu = relu;
    const bool tn = sa0 == 1 && sb1 == 1 && K > 0 && sa1 >= M && sb0 >= N && tn_pays(M, N, K);   // both operands along their rows
    static_assert(kTnK == kBK, "one rounding of the slices serves both kernels");
    g.slices = K > 0 ? (tn ? tn_row_slices(M, N, K) : sgemm_slices(M, N, K)) : 1;
    g.k_slice = ((K + g.slices - 1) / g.slices + kBK - 1) / kBK * kBK;
    if (g.k_slice < kBK) g.k_slice = kBK;
    g.slices = (int)((K + g.k_slice - 1) / g.k_slice);
    if (g.slices < 1) g.slices = 1;
    if (g.slices > 1) {
        const size_t need = (size_t)g.slices * (size_t)M * (size_t)N * sizeof(float);
        JG_CHECK_ARG(workspace && workspace_bytes >= need, JG_EWORKSPACE, "gemm_f32: workspace %zu < %zu", workspace_bytes, need);
        g.c = static_cast<float*>(workspace);
    } else {
        g.c = c;
    }
    if (tn) {
        switch (tn_cols(N)) {
            case 1: launch_tn<1>(g, st); break;
            case 2: launch_tn<2>(g, st); break;
            case 3: launch_tn<3>(g, st); break;
            case 4: launch_tn<4>(g, st); break;
            default: launch_tn<8>(g, st); break;
        }
    } else {
        dim3 grid((unsigned)((M + kBM - 1) / kBM), (unsigned)((N + kBN - 1) / kBN), (unsigned)g.slices);
        sgemm_kernel<<<grid, 256, 0, st>>>(g);
    }
    JG_LAUNCH_CHECK();
    return g.slices > 1 ? launch_reduce(c, static_cast<const float*>(workspace), M, N, ldc, g.slices, bias, relu, st) : JG_OK;
}

}  // extern "C"
