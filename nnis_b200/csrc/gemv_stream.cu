// Decode projections with many output features (gate/up, a mixer's stacked projections) of at most 16 rows:
// y[M, N] = x[M, K] . W[N, K]^T, x as it is, where W does not fit the SMs' shared memory.
//
// gemv_kernel.cuh gives a warp eight output features over all of K.  With K from 1,024 on that is a chain of chunks of 512
// columns a warp, two in flight, and whole units to 1,184 warps: 1,408 units of a gate/up product leave half of the warps
// idle for half of the time (2.6 TB/s).  Here a CTA takes a unit of eight output features at a time and its eight warps
// share K: x stays in the registers of their products for all units (as in gemv_rowtile.cu, a lane's four consecutive
// columns standing for the column pairs of the tile), and a unit costs a warp K / 128 products from shared memory.  The
// units' rows come whole by bulk copies into a ring, the first of them before the wait; a stage is asked for again as soon
// as the partial sums of its unit lie in shared memory, where one warp adds them in order and runs the epilogue while
// the others go on.
// What bounds it: the weights' way from memory.  M x N x K in us one after another in a graph, the kernel whose CTAs hold
// all rows -> here: gated 8 x 11,264 x 2,048 14.2 -> 9.0 (46 MB, 5.1 TB/s), 16 rows 14.4 -> 11.0, 8 x 16,384 x 3,072 30.3 -> 21.5;
// storing 8 x 6,144 x 2,048 8.0 -> 5.9, 8 x 12,288 x 2,560 23.9 -> 12.9, 8 x 2,400 x 2,048 7.1 -> 4.1.
#include "gemv_kernel.cuh"

namespace nnis {

constexpr int kStreamWarps = 8;
constexpr int kStreamStages = 3;

// elements between rows of W in shared memory: 32 bytes off a multiple of 128 (see rowtile_w_stride)
__host__ __device__ constexpr int stream_w_stride(int K) { return K + ((16 - K % 64) + 64) % 64; }

template <int EPI, int STEPS>
__global__ void __launch_bounds__(kStreamWarps * 32)
gemv_stream_kernel(GemvArgs a) {
    constexpr int WARPS = kStreamWarps, S = kStreamStages;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[S];
    __shared__ float red[2][WARPS][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    trace_mark(a.trace, 0);
    const int K = a.K, KPW = stream_w_stride(K), n_units = a.N >> 3;
    bf16* ws = reinterpret_cast<bf16*>(smem_raw);  // [S][8, KPW]
    const int steps = K >> 4, per_warp = (steps + WARPS - 1) / WARPS;
    const int k_begin = min(steps, warp * per_warp) * 16, k_end = min(steps, (warp + 1) * per_warp) * 16;
    const int mine = n_units > (int)blockIdx.x ? (n_units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    // the rows of this CTA's unit number i; a whole warp calls it
    auto ask = [&](int i) {
        const int unit = blockIdx.x + i * gridDim.x, s = i % S;
        if (lane == 0) mbar_expect_tx(&full[s], 8u * (uint32_t)K * 2u);
        __syncwarp();
        if (lane < 8)
            bulk_load(ws + ((size_t)s * 8 + lane) * KPW, a.w + (size_t)unit_row<EPI>(a, unit, lane) * K, (uint32_t)K * 2u,
                      &full[s]);
    };
    if (warp == 0) {
        if (lane == 0) {
            for (int s = 0; s < S; ++s) mbar_init(&full[s], 1);
            mbar_fence_init();
        }
        __syncwarp();
        for (int i = 0; i < S && i < mine; ++i) ask(i);
    }
    __syncthreads();  // every warp sees the barriers initialised
    pdl_wait();
    pdl_launch_dependents();
    trace_mark(a.trace, 2);
    trace_mark(a.trace, 3);

    uint32_t ax[STEPS][4];
    {
        const int g = lane >> 2, t4 = (lane & 3) * 4;
        const bf16* x0 = a.x + (size_t)g * K + k_begin + t4;
        const bf16* x1 = x0 + (size_t)8 * K;
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const bool in_k = k_begin + s * 16 < k_end;
            const uint2 zero = make_uint2(0u, 0u);
            const uint2 va = in_k && g < a.M ? *reinterpret_cast<const uint2*>(x0 + s * 16) : zero;
            const uint2 vb = in_k && g + 8 < a.M ? *reinterpret_cast<const uint2*>(x1 + s * 16) : zero;
            ax[s][0] = va.x;
            ax[s][1] = vb.x;
            ax[s][2] = va.y;
            ax[s][3] = vb.y;
        }
    }
    trace_mark(a.trace, 4);
    trace_mark(a.trace, 5);
    bool arrived = true;
    float best_v[2] = {0.f, 0.f};
    int best_i[2] = {-1, -1};
    EpiTile pre;
    for (int i = 0; i < mine; ++i) {
        const int s = i % S, buf = i & 1;
        // (a wait that runs out is flagged; the CTA goes on through its barriers)
        arrived = mbar_wait(&full[s], (uint32_t)(i / S) & 1u) && arrived;
        const bf16* b_ptr = ws + ((size_t)s * 8 + (lane >> 2)) * KPW + (lane & 3) * 4 + k_begin;
        float acc[2][4] = {};  // two chains of products
#pragma unroll
        for (int k = 0; k < STEPS; ++k)
            if (k_begin + k * 16 < k_end) {
                const uint2 bw = *reinterpret_cast<const uint2*>(b_ptr + k * 16);
                mma_bf16(acc[k & 1], ax[k], bw.x, bw.y);
            }
#pragma unroll
        for (int e = 0; e < 4; ++e) red[buf][warp][e][lane] = acc[0][e] + acc[1][e];
        __syncthreads();  // (also: the sums of unit i - 2, in the same place, have been read before unit i - 1's barrier)
        const int finisher = i % WARPS;
        if (warp == finisher) {
            if (i + S < mine) ask(i + S);
            float sum[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v = red[buf][0][e][lane];
#pragma unroll
                for (int w = 1; w < WARPS; ++w) v += red[buf][w][e][lane];
                sum[e] = v;
            }
            epi_finish<EPI>(a, blockIdx.x + i * gridDim.x, 0, lane, sum, pre, false, best_v, best_i);
        }
    }
    trace_mark(a.trace, 6);
    trace_mark(a.trace, 7);
    if (!arrived && lane == 0 && a.status) atomicExch(a.status, 2);
    trace_mark(a.trace, 1);
}

// Whether this kernel takes a product: one tile of rows, K in steps of 16 whose shares of x fit a warp's registers, and
// units for two CTAs an SM (with fewer, or a K below 1,024, the launches whose CTAs are all resident hold W at once:
// gated 8 x 5,632 x 1,024 4.0 there).
bool gemv_stream_takes(int M, int N, int K, int epilogue, int pro, int sm_count) {
    const int sms = sm_count > 0 ? sm_count : 148;
    return M > 0 && M <= 16 && K % 16 == 0 && K >= 1024 && K <= 24 * 16 * kStreamWarps && N % 8 == 0 && N / 8 >= 2 * sms &&
           pro == PRO_PLAIN && (epilogue == EPI_STORE || epilogue == EPI_STORE_F32 || epilogue == EPI_GATED);
}

template <int EPI, int STEPS>
static int launch_stream(const GemvArgs& a, int sms, bool pdl, cudaStream_t stream) {
    auto kernel = gemv_stream_kernel<EPI, STEPS>;
    const size_t smem = (size_t)kStreamStages * 8 * stream_w_stride(a.K) * sizeof(bf16);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    const int fit = smem <= 105 * 1024 ? 2 : 1;
    cfg.gridDim = dim3((unsigned)(a.N / 8 < sms * fit ? a.N / 8 : sms * fit));
    cfg.blockDim = dim3(kStreamWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

int gemv_launch_stream(const GemvArgs& a, int epi, int sm_count, bool pdl, cudaStream_t stream) {
    const int sms = sm_count > 0 ? sm_count : 148;
    const int steps = (a.K / 16 + kStreamWarps - 1) / kStreamWarps;
#define NNIS_STREAM(EPI) \
    return steps <= 12 ? launch_stream<EPI, 12>(a, sms, pdl, stream) \
         : steps <= 16 ? launch_stream<EPI, 16>(a, sms, pdl, stream) : launch_stream<EPI, 24>(a, sms, pdl, stream)
    if (epi == EPI_STORE) { NNIS_STREAM(EPI_STORE); }
    if (epi == EPI_STORE_F32) { NNIS_STREAM(EPI_STORE_F32); }
    if (epi == EPI_GATED) { NNIS_STREAM(EPI_GATED); }
#undef NNIS_STREAM
    return NNIS_ERR_UNSUPPORTED;
}

}  // namespace nnis
