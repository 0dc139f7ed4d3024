// Latent attention of single tokens (bfloat16): every row of the step is one token, and a CTA works 16 of its heads over
// a slice of its keys.
//
// The kernel of prompts (attention_latent_mma.cu) stacks (token, head) pairs into 64 or 128 rows and gives each warp 16
// of them: a token of 16 heads leaves three warps of four without rows, and the fourth multiplies a page's scores and
// values alone, one after another (8 tokens x 16 heads of 512 + 64 over 2,048 keys: 24.5 us).  Here the eight warps share
// a page: each takes eight of its keys for the scores, two of the 16 rows for the softmax (which meets in shared memory)
// and every eighth tile of 16 values for the output, whose sums it keeps in registers.  Pages come by TMA, a copy for 64
// of a row's values (boxes of 64 rows of 128 bytes in the 128-byte swizzle, so that eight rows meet no bank twice; the
// queries' rows are padded by 16 bytes instead), all that the ring holds before the wait for the kernel before: only the
// row of this step's token and the queries are fetched after it.  Rows that the token does not see are zero, whatever the
// page holds there.  What bounds it: a chain of few products and three barriers a page, and the slices' way into the
// merge.  16 heads of 512 + 64, merge included, in us in a graph, the kernel of prompts -> here: 8 tokens over 2,048 keys
// in 16 slices 28.8 -> 15.9, over 512 in 8 17.2 -> 10.8; one token over 2,048 26.9 -> 14.2; 32 tokens over 512 in 4 27.3
// -> 14.0; a page of a slice 8 -> 2.6.  8 heads of 256 + 32, 8 tokens over 2,048 keys in 16: 18.4 -> 10.2.
#include "attention_merge.cuh"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kLdPage = 64, kLdRows = 16, kLdWarps = 8;
constexpr int kLdTiles = 5;  // tiles of 16 values of a warp: dv <= 640

constexpr int kLdBox = kLdPage * 128;  // bytes of a box: 64 rows of 64 values, 128-byte swizzle

__host__ __device__ constexpr int latent_decode_stride(int dk) { return dk + 8; }  // of the queries' rows, in elements
__host__ __device__ constexpr int latent_decode_boxes(int dk) { return (dk + 63) / 64; }

// 16-byte chunk `chunk` of row `row` of a page
__device__ __forceinline__ unsigned char* page_chunk(unsigned char* page, int row, int chunk) {
    return page + (size_t)(chunk >> 3) * kLdBox + row * 128 + (((chunk & 7) ^ (row & 7)) << 4);
}

template <int STAGES>
__global__ void __launch_bounds__(kLdWarps * 32)
latent_decode_kernel(const __grid_constant__ CUtensorMap map, const bf16* __restrict__ q, const bf16* __restrict__ cache,
                     const int* __restrict__ token_pos, const int* __restrict__ token_seq,
                     const int* __restrict__ page_table, int table_cols,
                     bf16* __restrict__ out, float* __restrict__ partial, int heads, int dk, int dv, int head_tiles,
                     float scale, int n_splits, int window, const float* __restrict__ gate,
                     const float* __restrict__ sink, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[STAGES];
    __shared__ float s_s[kLdRows][kLdPage + 4];
    __shared__ __align__(16) bf16 p_s[kLdRows][kLdPage + 8];
    __shared__ float alpha_s[kLdRows], m_s[kLdRows], l_s[kLdRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int KP = latent_decode_stride(dk);
    const int boxes = latent_decode_boxes(dk);
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    bf16* q_s = reinterpret_cast<bf16*>(ring + (size_t)STAGES * boxes * kLdBox);  // [16, KP]
    const int n = blockIdx.x / head_tiles, h0 = (blockIdx.x - n * head_tiles) * kLdRows;
    const int rows = min(kLdRows, heads - h0), split = blockIdx.y;
    const int pos = token_pos[n];
    if (pos < 0) {  // (a padding row: the merge and the projections after it read nothing of it)
        pdl_wait();  // (a grid of such rows alone must not be over before the kernel ahead, which later ones count on)
        return;
    }
    const int lo = window > 0 ? max(0, pos - window + 1) : 0, hi = pos + 1;  // keys that the token sees
    const int seen_page = lo / kLdPage, end_page = (hi - 1) / kLdPage + 1;
    const int per = (end_page - seen_page + n_splits - 1) / n_splits;
    const int first_page = seen_page + split * per;
    const int n_pages = max(0, min(end_page, first_page + per) - first_page);
    const int* table = page_table + (size_t)token_seq[n] * table_cols;
    auto first_row = [&](int it) { return max(0, lo - (first_page + it) * kLdPage); };
    auto end_row = [&](int it) { return min(kLdPage, hi - (first_page + it) * kLdPage); };
    auto ask = [&](int it) {  // one thread
        unsigned char* dst = ring + (size_t)(it % STAGES) * boxes * kLdBox;
        const int row = table[first_page + it] * kLdPage;
        mbar_expect_tx(&full[it % STAGES], (uint32_t)(boxes * kLdBox));
        for (int b = 0; b < boxes; ++b) tma_load_2d(dst + (size_t)b * kLdBox, &map, b * 64, row, &full[it % STAGES]);
    };
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map);
        for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
        for (int it = 0; it < STAGES && it < n_pages; ++it) ask(it);
    }
    // the eight columns after a row's values count as zeros where dk is no multiple of 16 (a page's come as zeros)
    if (threadIdx.x < kLdRows) *reinterpret_cast<uint4*>(q_s + (size_t)threadIdx.x * KP + dk) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    const int chunks = dk >> 3;
    for (int c = threadIdx.x; c < kLdRows * chunks; c += kLdWarps * 32) {
        const int row = c / chunks, chunk = c - row * chunks;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (row < rows) v = *reinterpret_cast<const uint4*>(q + ((size_t)n * heads + h0 + row) * dk + chunk * 8);
        *reinterpret_cast<uint4*>(q_s + (size_t)row * KP + chunk * 8) = v;
    }
    const int r_lo = lane >> 2, c_lo = (lane & 3) * 2;
    const int k_steps = (dk + 15) >> 4, v_tiles = dv >> 4;
    const float sc = scale * kLog2e;
    // rows 2 warp and 2 warp + 1 of the softmax are this warp's
    float m_run[2], l_run[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int row = warp * 2 + j;
        const bool has_sink = sink && split == 0 && row < rows;  // a score without a key and without a value
        m_run[j] = has_sink ? sink[h0 + row] * kLog2e : -INFINITY;
        l_run[j] = has_sink ? 1.f : 0.f;
    }
    float o[kLdTiles][2][4];
#pragma unroll
    for (int t = 0; t < kLdTiles; ++t)
#pragma unroll
        for (int e = 0; e < 8; ++e) o[t][e >> 2][e & 3] = 0.f;
    bool arrived = true;
    __syncthreads();
    for (int it = 0; it < n_pages; ++it) {
        const int s = it % STAGES;
        unsigned char* kt = ring + (size_t)s * boxes * kLdBox;
        // (a wait that runs out is flagged; the CTA goes on through its barriers)
        arrived = mbar_wait(&full[s], (uint32_t)(it / STAGES) & 1u) && arrived;
        const int r0 = first_row(it), r1 = end_row(it), page_end = (first_page + it) * kLdPage + r1;
        if (r0 > 0 || r1 < kLdPage || page_end == hi) {
            for (int c = threadIdx.x; c < kLdPage * chunks; c += kLdWarps * 32) {
                const int row = c / chunks, chunk = c - row * chunks;
                uint4* at = reinterpret_cast<uint4*>(page_chunk(kt, row, chunk));
                if (row < r0 || row >= r1) *at = make_uint4(0, 0, 0, 0);
                else if (page_end == hi && row == r1 - 1)  // this step's row: written by the kernels just before
                    *at = *reinterpret_cast<const uint4*>(cache + ((size_t)table[first_page + it] * kLdPage + row) * dk + chunk * 8);
            }
            // (a window's first page is one that the ring asks for again: these stores come before the copies over them)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
        // scores of keys 8 warp .. 8 warp + 7
        float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
        const bf16* qp = q_s + (size_t)(lane & 15) * KP + (lane >> 4) * 8;
        int ks = 0;
#pragma unroll 3
        for (; ks + 2 <= k_steps; ks += 2) {
            uint32_t qa0[4], qa1[4], b[4];
            ldmatrix_x4(qa0, qp + ks * 16);
            ldmatrix_x4(qa1, qp + ks * 16 + 16);
            ldmatrix_x4(b, page_chunk(kt, warp * 8 + (lane & 7), ks * 2 + (lane >> 3)));
            mma_bf16(a0, qa0, b[0], b[1]);
            mma_bf16(a1, qa1, b[2], b[3]);
        }
        if (ks < k_steps) {
            uint32_t qa0[4], b[4];
            ldmatrix_x4(qa0, qp + ks * 16);
            ldmatrix_x4(b, page_chunk(kt, warp * 8 + (lane & 7), ks * 2 + ((lane >> 3) & 1)));
            mma_bf16(a0, qa0, b[0], b[1]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int key = warp * 8 + c_lo + (e & 1);
            s_s[r_lo + (e >> 1) * 8][key] = key >= r0 && key < r1 ? (a0[e] + a1[e]) * sc : -INFINITY;
        }
        __syncthreads();
        // (every warp is through with the page before this one)
        if (threadIdx.x == 0 && it > 0 && it - 1 + STAGES < n_pages) ask(it - 1 + STAGES);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int row = warp * 2 + j;
            const float v0 = s_s[row][lane], v1 = s_s[row][lane + 32];
            const float mn = fmaxf(m_run[j], warp_max(fmaxf(v0, v1)));
            const float base = mn == -INFINITY ? 0.f : mn;
            const float alpha = exp2f(m_run[j] - base), p0 = exp2f(v0 - base), p1 = exp2f(v1 - base);
            m_run[j] = mn;
            l_run[j] = l_run[j] * alpha + warp_sum(p0 + p1);
            p_s[row][lane] = __float2bfloat16_rn(p0);
            p_s[row][lane + 32] = __float2bfloat16_rn(p1);
            if (lane == 0) alpha_s[row] = alpha;
        }
        __syncthreads();
        const float al = alpha_s[r_lo], ah = alpha_s[r_lo + 8];
        uint32_t pa[kLdPage / 16][4];
#pragma unroll
        for (int k = 0; k < kLdPage / 16; ++k) ldmatrix_x4(pa[k], &p_s[lane & 15][k * 16 + (lane >> 4) * 8]);
#pragma unroll
        for (int t = 0; t < kLdTiles; ++t) {
            const int tile = warp + t * kLdWarps;
            if (tile >= v_tiles) break;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                o[t][half][0] *= al;
                o[t][half][1] *= al;
                o[t][half][2] *= ah;
                o[t][half][3] *= ah;
            }
#pragma unroll
            for (int k = 0; k < kLdPage / 16; ++k) {
                uint32_t b[4];
                ldmatrix_x4_trans(b, page_chunk(kt, k * 16 + (lane & 15), tile * 2 + (lane >> 4)));
                mma_bf16(o[t][0], pa[k], b[0], b[1]);
                mma_bf16(o[t][1], pa[k], b[2], b[3]);
            }
        }
    }
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            m_s[warp * 2 + j] = m_run[j];
            l_s[warp * 2 + j] = l_run[j];
        }
    if (!arrived && lane == 0 && status) atomicExch(status, 2);
    __syncthreads();
    const size_t row_base = (size_t)n * heads + h0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = r_lo + h * 8;
        if (row >= rows) continue;
        const float l = l_s[row];
        if (n_splits == 1) {
            float inv = l > 0.f ? 1.0f / l : 0.f;
            if (gate) inv *= gate[row_base + row];
#pragma unroll
            for (int t = 0; t < kLdTiles; ++t) {
                const int tile = warp + t * kLdWarps;
                if (tile >= v_tiles) break;
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<uint32_t*>(out + (row_base + row) * dv + tile * 16 + half * 8 + c_lo) =
                        pack_bf16(o[t][half][h * 2] * inv, o[t][half][h * 2 + 1] * inv);
            }
        } else {
            // records in natural-logarithm terms: o and l are relative to exp(m)
            float* rec = partial + ((row_base + row) * n_splits + split) * (size_t)(dv + 2);
            if (warp == 0 && (lane & 3) == 0) {
                rec[0] = l > 0.f ? m_s[row] * 0.6931471805599453f : 0.f;
                rec[1] = l;
            }
#pragma unroll
            for (int t = 0; t < kLdTiles; ++t) {
                const int tile = warp + t * kLdWarps;
                if (tile >= v_tiles) break;
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<float2*>(rec + 2 + tile * 16 + half * 8 + c_lo) =
                        make_float2(o[t][half][h * 2], o[t][half][h * 2 + 1]);
            }
        }
    }
}

static size_t latent_decode_smem(int dk, int stages) {
    return (size_t)stages * latent_decode_boxes(dk) * kLdBox + (size_t)kLdRows * latent_decode_stride(dk) * sizeof(bf16) + 1024;
}

}  // namespace nnis

using namespace nnis;

// Whether this kernel runs a step of single tokens of these sizes: rows of 16-byte pieces, values in tiles of 16, two pages
// in shared memory.  Up to two tiles of heads: each fetches the pages again (32 heads, 8 tokens over 2,048 keys: 43.9 -> 19.0
// us in 8 slices; 64 would be level with the kernel of prompts, whose 64 rows share a page).
NNIS_API int nnis_attention_latent_decode_takes(int heads, int dk, int dv, int page_size) {
    return heads > 0 && heads <= 32 && dk > 0 && dk % 8 == 0 && dv > 0 && dv % 16 == 0 && dv <= dk &&
           dv <= 16 * kLdTiles * kLdWarps && page_size == kLdPage && latent_decode_smem(dk, 2) <= 220 * 1024;
}

// Arguments as nnis_attention_latent_mma without tiles; `partial` starts on an 8-byte boundary.
NNIS_API int nnis_attention_latent_decode(const void* q, const void* cache, const int* token_pos, const int* token_seq,
                                          const int* page_table, int table_cols, void* out, float* partial, int n_tokens,
                                          int heads, int dk, int dv, int pages, int page_size, float scale, int n_splits,
                                          int window, const float* gate, const float* sink, int* status,
                                          cudaStream_t stream) {
    if (pages <= 0 || n_tokens <= 0 || table_cols <= 0 || n_splits <= 0 || window < 0 || !q || !cache || !out || !page_table ||
        !token_pos || !token_seq)
        return NNIS_ERR_ARGUMENT;
    if (!nnis_attention_latent_decode_takes(heads, dk, dv, page_size) || n_splits > 64) return NNIS_ERR_UNSUPPORTED;
    if (n_splits > 1 && !partial) return NNIS_ERR_ARGUMENT;
    if (((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) % 16 || (uintptr_t)partial % 8) return NNIS_ERR_ALIGNMENT;
    const int head_tiles = (heads + kLdRows - 1) / kLdRows;
    CUtensorMap map;
    if (!make_map(&map, cache, (long long)pages * kLdPage, dk, kLdPage)) return NNIS_ERR_UNSUPPORTED;
    // (as many pages in flight as leave two CTAs to an SM, two at least)
    const int stages = latent_decode_smem(dk, 4) <= 100 * 1024 ? 4 : latent_decode_smem(dk, 3) <= 100 * 1024 ? 3 : 2;
    const size_t smem = latent_decode_smem(dk, stages);
    auto kernel = stages == 4 ? latent_decode_kernel<4> : stages == 3 ? latent_decode_kernel<3> : latent_decode_kernel<2>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    e = launch_dependent(kernel, dim3((unsigned)(n_tokens * head_tiles), (unsigned)n_splits), kLdWarps * 32, smem, stream,
                         map, (const bf16*)q, (const bf16*)cache, token_pos, token_seq, page_table, table_cols, (bf16*)out, partial,
                         heads, dk, dv, head_tiles, scale, n_splits, window, gate, sink, status);
    if (e != cudaSuccess) return (int)e;
    if (n_splits > 1)
        e = launch_merge<bf16>(partial, (bf16*)out, (size_t)n_tokens * heads, dv, n_splits, gate, stream);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
