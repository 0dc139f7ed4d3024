// Matrix products on the CUDA cores: C[M,N] (op)= A[M,K] . W[N,K]^T + bias.
// W is stored [out, in] row-major as the checkpoint has it, so both operands
// run along K.  Operands are float32 or bfloat16; products are accumulated in
// float32 with fmaf, never through a reduced-precision tensor-core mode.  These
// are the float32 path of single tokens and of the shapes and addresses that
// gemm_split_f32.cu does not take, and the fallback of the bfloat16 path for
// shapes that the tcgen05 kernel refuses.
//
// Output modes: 0 store in the operand dtype, 1 store float32, 2 add to a
// float32 destination (the residual stream).
// NNIS: crates/nnis-kernels/src/gemm.rs:16-64 (tiled product),
// crates/nnis-kernels/src/gemv.rs:45-61 (one-token projection).
#include "common.cuh"
#include "fma_pairs.cuh"

namespace nnis {

template <typename T, int MODE>
__device__ __forceinline__ void emit(void* C, size_t idx, float v) {
    if (MODE == 0) reinterpret_cast<T*>(C)[idx] = from_float<T>(v);
    else if (MODE == 1) reinterpret_cast<float*>(C)[idx] = v;
    else reinterpret_cast<float*>(C)[idx] += v;
}

// ---- 64 x 64 tile, 256 threads: four groups of 64 threads share K, 8 x 8 outputs per thread ----
// A slab of 32 columns of K at a time, two in shared memory; group g multiplies columns 8 g .. 8 g + 7 of every
// slab and the four sums meet at the end (in the order of the groups: the same bits every time).  Splitting K inside
// the CTA is what lets the tile be small enough for a width of 576 (144 tiles at 1,024 rows) and still have eight
// warps.  A slab comes as whole 128-byte lines and is turned on its way into shared memory; groups of four rows are
// put at group ^ (column / 4), so that neither the turned stores nor the reads meet a bank twice.
// What bounds it: the multiply-add pipe (busy 58 % of the time under ncu) and, level with it, shared memory (52 %: an
// 8 x 8 tile of outputs reads four 16-byte words for 64 multiply-adds), with a last wave of tiles that is not full.
// 1,024 rows on a B200, before (4 x 4 outputs a thread, two words for 16, every slab waited for) and now:
// N x K = 3,072 x 576 130 -> 101 us (36 TFLOP/s), 960 x 576 52 -> 37, 576 x 576 33 -> 24, 576 x 1,536 80 -> 57.
// Level or slower: slabs left as they lie and brought three ahead by asynchronous copies, with single multiply-adds
// (112 us: one instruction for two is what the schedulers are short of); A kept twice side by side to save the moves
// (155 us, with rows fetched 32 bytes at a time).
template <typename T, bool VEC>
__device__ __forceinline__ float4 slab_load(const T* __restrict__ p, int row, int rows, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    p += (size_t)row * K;
    if (VEC) {
        if (k < K) v = load4(p + k);
    } else {
        if (k < K) v.x = to_float(p[k]);
        if (k + 1 < K) v.y = to_float(p[k + 1]);
        if (k + 2 < K) v.z = to_float(p[k + 2]);
        if (k + 3 < K) v.w = to_float(p[k + 3]);
    }
    return v;
}

constexpr int kSlabM = 64, kSlabN = 64, kSlabK = 32;
constexpr int kSlabSmem = 4 * 32 * 64 * 8;  // the sums of the four groups; the slabs (32 KB) lie in the same place
static_assert(2 * kSlabK * (kSlabM + kSlabN) * 4 <= kSlabSmem, "slabs fit where the sums go");

template <typename T, int MODE, bool VEC>
__global__ void __launch_bounds__(256, 2)
gemm_slab_kernel(const T* __restrict__ A, const T* __restrict__ W, const float* __restrict__ bias,
                 void* __restrict__ C, int M, int N, int K) {
    extern __shared__ __align__(16) unsigned char slab_smem[];
    float* As = reinterpret_cast<float*>(slab_smem);  // [2][32][64]
    float* Ws = As + 2 * kSlabK * kSlabM;             // [2][32][64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * kSlabM, n0 = blockIdx.x * kSlabN;
    // a warp brings four rows of 32 columns at a time, eight rows in all
    const int load_row = warp * 8 + (lane >> 3), load_k = (lane & 7) * 4;
    float4 ra[2], rw[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            ra[j] = slab_load<T, VEC>(A, m0 + load_row + 4 * j, M, k0 + load_k, K);
            rw[j] = slab_load<T, VEC>(W, n0 + load_row + 4 * j, N, k0 + load_k, K);
        }
    };
    auto keep = [&](int buf) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int at = (buf * kSlabK + load_k) * 64 + (((warp * 2 + j) ^ (lane & 7)) << 2) + (lane >> 3);
            As[at] = ra[j].x;
            As[at + 64] = ra[j].y;
            As[at + 128] = ra[j].z;
            As[at + 192] = ra[j].w;
            Ws[at] = rw[j].x;
            Ws[at + 64] = rw[j].y;
            Ws[at + 128] = rw[j].z;
            Ws[at + 192] = rw[j].w;
        }
    };
    const int group = tid >> 6, t = tid & 63, tx = t & 7, ty = t >> 3;
    unsigned long long acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    const int slabs = (K + kSlabK - 1) / kSlabK;
    fetch(0);
    keep(0);
    __syncthreads();
    for (int s = 0; s < slabs; ++s) {
        if (s + 1 < slabs) fetch((s + 1) * kSlabK);
        const float* a0 = As + ((s & 1) * kSlabK + group * 8) * 64;
        const float* w0 = Ws + ((s & 1) * kSlabK + group * 8) * 64;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int turn = (group * 2 + (k >> 2)) & 7;  // column / 4 within the slab
            const int ao = k * 64 + ((ty ^ turn) << 2), wo = k * 64 + ((tx ^ turn) << 2);
            const float4 al = load4(a0 + ao), ah = load4(a0 + ao + 32);
            ulonglong2 wv[2];
            wv[0] = *reinterpret_cast<const ulonglong2*>(w0 + wo);
            wv[1] = *reinterpret_cast<const ulonglong2*>(w0 + wo + 32);
            const float av[8] = {al.x, al.y, al.z, al.w, ah.x, ah.y, ah.z, ah.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long a = both(av[i]);
                fma2(acc[i][0], a, wv[0].x);
                fma2(acc[i][1], a, wv[0].y);
                fma2(acc[i][2], a, wv[1].x);
                fma2(acc[i][3], a, wv[1].y);
            }
        }
        if (s + 1 < slabs) keep((s + 1) & 1);  // (last read before the barrier that ended slab s - 1)
        __syncthreads();
    }
    // the groups' sums: group g finishes rows 2 g and 2 g + 1 of every thread's eight
    unsigned long long* sums = reinterpret_cast<unsigned long long*>(slab_smem);  // [4 groups][32 pairs][64 threads]
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[(group * 32 + i * 4 + j) * 64 + t] = acc[i][j];
    __syncthreads();
    const bool by_four = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int i = group * 2 + r, m = m0 + (i < 4 ? 0 : 32) + ty * 4 + (i & 3);
        if (m >= M) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float v[4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const float2 x = reinterpret_cast<const float2*>(sums)[(g * 32 + i * 4 + half * 2 + p) * 64 + t];
                    sum.x += x.x;
                    sum.y += x.y;
                }
                v[2 * p] = sum.x;
                v[2 * p + 1] = sum.y;
            }
            const int n = n0 + half * 32 + tx * 4;
            const size_t at = (size_t)m * N + n;
            if (by_four && n < N) {
                float4 o = make_float4(v[0], v[1], v[2], v[3]);
                if (bias) o = make_float4(o.x + bias[n], o.y + bias[n + 1], o.z + bias[n + 2], o.w + bias[n + 3]);
                if (MODE == 0) store4(reinterpret_cast<T*>(C) + at, o);
                else if (MODE == 1) store4(reinterpret_cast<float*>(C) + at, o);
                else {
                    const float4 c = load4(reinterpret_cast<const float*>(C) + at);
                    store4(reinterpret_cast<float*>(C) + at, make_float4(c.x + o.x, c.y + o.y, c.z + o.z, c.w + o.w));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < N) emit<T, MODE>(C, at + e, v[e] + (bias ? bias[n + e] : 0.f));
            }
        }
    }
}

// ---- few rows (decoding): one warp per output column, MT rows at a time -----
template <typename T, int MT, int MODE, bool VEC>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const T* __restrict__ A, const T* __restrict__ W, const float* __restrict__ bias,
                 void* __restrict__ C, int M, int N, int K) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int n = blockIdx.x * 8 + warp;
    int m0 = blockIdx.y * MT;
    if (n >= N) return;
    float acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0.f;
    const T* wrow = W + (size_t)n * K;
    if (VEC) {
        for (int k = lane * 4; k < K; k += 128) {
            float4 w = load4(wrow + k);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                if (m0 + i < M) {
                    float4 a = load4(A + (size_t)(m0 + i) * K + k);
                    acc[i] = fmaf(a.x, w.x, acc[i]);
                    acc[i] = fmaf(a.y, w.y, acc[i]);
                    acc[i] = fmaf(a.z, w.z, acc[i]);
                    acc[i] = fmaf(a.w, w.w, acc[i]);
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            float w = to_float(wrow[k]);
#pragma unroll
            for (int i = 0; i < MT; ++i)
                if (m0 + i < M) acc[i] = fmaf(to_float(A[(size_t)(m0 + i) * K + k]), w, acc[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        float v = warp_sum(acc[i]);
        if (lane == 0 && m0 + i < M)
            emit<T, MODE>(C, (size_t)(m0 + i) * N + n, v + (bias ? bias[n] : 0.f));
    }
}

template <typename T, int MODE, bool VEC>
static int launch_mode(const T* A, const T* W, const float* bias, void* C, int M, int N, int K,
                       cudaStream_t stream) {
    if (M <= 16) {
        dim3 grid((N + 7) / 8, 1);
        if (M == 1) gemm_rows_kernel<T, 1, MODE, VEC><<<grid, 256, 0, stream>>>(A, W, bias, C, M, N, K);
        else if (M == 2) gemm_rows_kernel<T, 2, MODE, VEC><<<grid, 256, 0, stream>>>(A, W, bias, C, M, N, K);
        else if (M <= 4) gemm_rows_kernel<T, 4, MODE, VEC><<<grid, 256, 0, stream>>>(A, W, bias, C, M, N, K);
        else {
            grid.y = (M + 7) / 8;
            gemm_rows_kernel<T, 8, MODE, VEC><<<grid, 256, 0, stream>>>(A, W, bias, C, M, N, K);
        }
    } else {
        dim3 grid((N + kSlabN - 1) / kSlabN, (M + kSlabM - 1) / kSlabM);
        if (grid.y > 65535u) return NNIS_ERR_UNSUPPORTED;
        cudaError_t e = cudaFuncSetAttribute(gemm_slab_kernel<T, MODE, VEC>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmem);
        if (e != cudaSuccess) return (int)e;
        gemm_slab_kernel<T, MODE, VEC><<<grid, 256, kSlabSmem, stream>>>(A, W, bias, C, M, N, K);
    }
    NNIS_RETURN_LAUNCH();
}

template <typename T>
static int launch_type(const void* A, const void* W, const float* bias, void* C, int M, int N, int K,
                       int mode, cudaStream_t stream) {
    const T* a = (const T*)A;
    const T* w = (const T*)W;
    bool vec = (K % 4 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
#define NNIS_GEMM_CASE(MODE) \
    return vec ? launch_mode<T, MODE, true>(a, w, bias, C, M, N, K, stream) \
               : launch_mode<T, MODE, false>(a, w, bias, C, M, N, K, stream)
    switch (mode) {
        case 0: NNIS_GEMM_CASE(0);
        case 1: NNIS_GEMM_CASE(1);
        case 2: NNIS_GEMM_CASE(2);
        default: return NNIS_ERR_ARGUMENT;
    }
#undef NNIS_GEMM_CASE
}

}  // namespace nnis

NNIS_API int nnis_gemm_simt(const void* A, const void* W, const float* bias, void* C, int M, int N,
                            int K, int dtype, int mode, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || !A || !W || !C) return NNIS_ERR_ARGUMENT;
    if (dtype == NNIS_DTYPE_F32) return nnis::launch_type<float>(A, W, bias, C, M, N, K, mode, stream);
    if (dtype == NNIS_DTYPE_BF16) return nnis::launch_type<nnis::bf16>(A, W, bias, C, M, N, K, mode, stream);
    return NNIS_ERR_UNSUPPORTED;
}
