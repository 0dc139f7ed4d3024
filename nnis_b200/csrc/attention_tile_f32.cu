// Prompt attention in true float32 over the paged cache, for head sizes that attention_split_f32.cu does not take and, with
// heads of 64, for steps of many prompts that see one page each: 64 consecutive queries of a sequence and one query head
// per CTA, a page of 64 keys at a time.  Both products are tiled in registers (4 queries x 4 keys, then 4 queries
// x 4 or 8 output values a thread), so a key or value fetched once serves 64 queries; the any-size kernel
// (attention_generic.cu), which this one takes prompts from, reads every key again for every query.  Scores,
// softmax and sums are float32 with fmaf and expf, never a reduced-precision product.  The key range of a tile may
// be split over several CTAs whose partial records (attention_generic.cu's) attn_merge_kernel puts together.
// What bounds it: the multiply-add pipe and the shared-memory reads beside it (three wavefronts for sixteen
// multiply-adds of a warp); the copies of a page are waited for, which the other two or three CTAs of the SM hide.
// Three prompts of 1,024 tokens together, 9 heads of 64, on a B200: 219 -> 61 us a layer, 11 us of it the merge.
#include <float.h>

#include "attention_merge.cuh"
#include "common.cuh"

namespace nnis {

constexpr int kTileRows = 64, kTileKeys = 64, kTileLd = 68;  // (rows of 68 floats: 16-byte aligned, no bank met twice)

// D: the head size rounded up to 64 or 128; d: the head size, a multiple of four
template <int D>
__global__ void __launch_bounds__(256)
attn_tile_f32_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ k_cache,
                     const float* __restrict__ v_cache, const int2* __restrict__ tiles,
                     const int* __restrict__ seq_first_row, const int* __restrict__ seq_start,
                     const int* __restrict__ seq_count, const int* __restrict__ page_table, int table_cols,
                     float* __restrict__ out, float* __restrict__ partial, int nq, int nkv, int d, int window,
                     float scale, int n_splits) {
    extern __shared__ __align__(16) float tile_smem[];
    float* qs = tile_smem;              // [d][68]: queries, their values down the rows
    float* ks = qs + D * kTileLd;       // [d][68]: a page's keys, the same way
    float* ps = ks + D * kTileLd;       // [64 keys][68]: softmax weights, a row per key
    float* vs = ps + kTileKeys * kTileLd;  // [64 keys][D]
    constexpr int C = D / 64;           // four output columns a thread, C times
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
    const int2 tile = tiles[blockIdx.x];
    const int seq = tile.x, q0 = tile.y, hq = blockIdx.y, hk = hq / (nq / nkv);
    const int rows = min(kTileRows, seq_count[seq] - q0);
    const int pos0 = seq_start[seq] + q0, row0 = seq_first_row[seq] + q0;
    const int* table = page_table + (size_t)seq * table_cols;
    const int lo = window > 0 ? max(0, pos0 - window + 1) : 0;
    const int first_page = lo / kTileKeys, all_pages = (pos0 + rows - 1) / kTileKeys - first_page + 1;
    const int per = (all_pages + n_splits - 1) / n_splits;
    const int p_begin = first_page + (int)blockIdx.z * per;
    const int p_end = min(first_page + all_pages, p_begin + per);

    // 16 rows x 8 columns a warp: rows are neighbours in shared memory
    const int lrow = (warp & 3) * 16 + (lane & 15), lcol = (warp >> 2) * 8 + (lane >> 4) * 4;
    for (int c = lcol; c < d; c += 16) {
        const float4 v = lrow < rows ? load4(q + (size_t)(row0 + lrow) * q_stride + (size_t)hq * d + c)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
        qs[c * kTileLd + lrow] = v.x;
        qs[(c + 1) * kTileLd + lrow] = v.y;
        qs[(c + 2) * kTileLd + lrow] = v.z;
        qs[(c + 3) * kTileLd + lrow] = v.w;
    }
    float m[4], l[4], acc[4][4 * C];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -FLT_MAX;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * C; ++c) acc[i][c] = 0.f;
    }
    for (int p = p_begin; p < p_end; ++p) {
        const size_t base = ((size_t)table[p] * nkv + hk) * kTileKeys * d;
        __syncthreads();  // the page before is done with
        for (int c = lcol; c < d; c += 16) {
            const float4 v = load4(k_cache + base + (size_t)lrow * d + c);
            ks[c * kTileLd + lrow] = v.x;
            ks[(c + 1) * kTileLd + lrow] = v.y;
            ks[(c + 2) * kTileLd + lrow] = v.z;
            ks[(c + 3) * kTileLd + lrow] = v.w;
        }
        for (int it = tid; it < kTileKeys * (D / 4); it += 256) {
            const int r = it / (D / 4), c = (it % (D / 4)) * 4;
            store4(vs + r * D + c, c < d ? load4(v_cache + base + (size_t)r * d + c) : make_float4(0.f, 0.f, 0.f, 0.f));
        }
        __syncthreads();
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 8
        for (int x = 0; x < d; ++x) {
            const float4 a = load4(qs + x * kTileLd + ty * 4), b = load4(ks + x * kTileLd + tx * 4);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = fmaf(av[i], bv[j], s[i][j]);
        }
        // softmax: a row's 64 scores lie with the sixteen threads of a half warp.  A slot of the page that no
        // token has filled may hold anything, so what is not visible is replaced before any arithmetic
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + ty * 4 + i;
            bool seen[4];
            float top = -FLT_MAX;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = p * kTileKeys + tx * 4 + j;
                seen[j] = t <= pos && (window <= 0 || pos - t < window);
                s[i][j] = seen[j] ? s[i][j] * scale : -FLT_MAX;
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m[i], top);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = seen[j] ? expf(s[i][j] - m_new) : 0.f;
                sum += s[i][j];
            }
            sum = half_warp_sum(sum);
            const float alpha = l[i] == 0.f ? 0.f : expf(m[i] - m_new);
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * C; ++c) acc[i][c] *= alpha;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            store4(ps + (j * 16 + tx) * kTileLd + ty * 4, make_float4(s[0][j], s[1][j], s[2][j], s[3][j]));
        __syncwarp();  // (a warp reads only the eight queries that it wrote)
        // (key 4 u + e is row 16 e + u of ps.)  On a page that not every query of the tile sees whole, a value row is
        // read only for the queries with a weight: a later token's, or what an empty slot holds, may be no number
        const bool edge = (p + 1) * kTileKeys - 1 > pos0 || (window > 0 && p * kTileKeys <= pos0 + rows - 1 - window);
        const int quads = edge ? (min(kTileKeys, pos0 + rows - p * kTileKeys) + 3) / 4 : kTileKeys / 4;
#pragma unroll 1
        for (int u = 0; u < quads; ++u) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 w = load4(ps + (e * 16 + u) * kTileLd + ty * 4);
                const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int h = 0; h < C; ++h) {
                    const float4 v = load4(vs + (u * 4 + e) * D + h * 64 + tx * 4);
                    if (!edge) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            acc[i][4 * h] = fmaf(wv[i], v.x, acc[i][4 * h]);
                            acc[i][4 * h + 1] = fmaf(wv[i], v.y, acc[i][4 * h + 1]);
                            acc[i][4 * h + 2] = fmaf(wv[i], v.z, acc[i][4 * h + 2]);
                            acc[i][4 * h + 3] = fmaf(wv[i], v.w, acc[i][4 * h + 3]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (wv[i] != 0.f) {
                                acc[i][4 * h] = fmaf(wv[i], v.x, acc[i][4 * h]);
                                acc[i][4 * h + 1] = fmaf(wv[i], v.y, acc[i][4 * h + 1]);
                                acc[i][4 * h + 2] = fmaf(wv[i], v.z, acc[i][4 * h + 2]);
                                acc[i][4 * h + 3] = fmaf(wv[i], v.w, acc[i][4 * h + 3]);
                            }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (r >= rows) continue;
        const size_t row = (size_t)(row0 + r) * nq + hq;
        if (n_splits == 1) {
            const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
#pragma unroll
            for (int h = 0; h < C; ++h) {
                const int c = h * 64 + tx * 4;
                if (c < d)
                    store4(out + row * d + c, make_float4(acc[i][4 * h] * inv, acc[i][4 * h + 1] * inv,
                                                          acc[i][4 * h + 2] * inv, acc[i][4 * h + 3] * inv));
            }
        } else {
            float* rec = partial + (row * n_splits + blockIdx.z) * (size_t)(d + 2);
            if (tx == 0) {
                rec[0] = m[i];
                rec[1] = l[i];
            }
#pragma unroll
            for (int h = 0; h < C; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (h * 64 + tx * 4 + e < d) rec[2 + h * 64 + tx * 4 + e] = acc[i][4 * h + e];
        }
    }
}

template <int D>
static int launch_tiles(const float* q, int q_stride, const float* k_cache, const float* v_cache, const int* tiles,
                        int n_tiles, const int* seq_first_row, const int* seq_start, const int* seq_count,
                        const int* page_table, int table_cols, float* out, float* partial, int nq, int nkv, int d,
                        int window, float scale, int n_splits, cudaStream_t stream) {
    const int smem = (2 * D * kTileLd + kTileKeys * kTileLd + kTileKeys * D) * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(attn_tile_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    attn_tile_f32_kernel<D><<<dim3(n_tiles, nq, n_splits), 256, smem, stream>>>(
        q, q_stride, k_cache, v_cache, reinterpret_cast<const int2*>(tiles), seq_first_row, seq_start, seq_count,
        page_table, table_cols, out, partial, nq, nkv, d, window, scale, n_splits);
    e = cudaGetLastError();
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

}  // namespace nnis

// float32 only, pages of 64 keys, head sizes up to 128 that are a multiple of four; else NNIS_ERR_UNSUPPORTED.
// `tiles`: int32 [n_tiles, 2] = (sequence of the batch, first query among this step's tokens of it), 64 queries each.
// Scratch: `partial` needs n_tokens * nq * n_splits * (d + 2) floats when n_splits > 1 and may be null otherwise.
NNIS_API int nnis_attention_tile_f32(const void* q, int q_stride, const void* k_cache, const void* v_cache,
                                     const int* tiles, int n_tiles, const int* seq_first_row, const int* seq_start,
                                     const int* seq_count, const int* page_table, int table_cols, void* out,
                                     float* partial, int n_tokens, int nq, int nkv, int d, int page_size, int window,
                                     float scale, int n_splits, cudaStream_t stream) {
    using namespace nnis;
    if (n_tiles <= 0 || n_tokens <= 0 || nq <= 0 || nkv <= 0 || nq % nkv || table_cols <= 0 || n_splits <= 0 ||
        window < 0 || !tiles || (n_splits > 1 && !partial))
        return NNIS_ERR_ARGUMENT;
    if (page_size != kTileKeys || d <= 0 || d % 4 || d > 128 || q_stride % 4 || nq > 65535 || n_splits > 64)
        return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) % 16 || (uintptr_t)tiles % 8)
        return NNIS_ERR_ALIGNMENT;
    int rc = (d <= 64 ? launch_tiles<64> : launch_tiles<128>)(
        (const float*)q, q_stride, (const float*)k_cache, (const float*)v_cache, tiles, n_tiles, seq_first_row,
        seq_start, seq_count, page_table, table_cols, (float*)out, partial, nq, nkv, d, window, scale, n_splits, stream);
    if (rc != NNIS_OK || n_splits == 1) return rc;
    const size_t rows = (size_t)n_tokens * nq;
    const cudaError_t e = launch_merge<float>(partial, (float*)out, rows, d, n_splits, nullptr, stream);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
