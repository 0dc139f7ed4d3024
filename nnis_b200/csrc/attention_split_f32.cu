// Prompt attention in float32 over the paged cache on the fifth-generation tensor cores, head size 64: 128 consecutive
// queries of a sequence and one query head per CTA, a page of 64 keys at a time.  Queries, keys, values and softmax weights
// enter both products as the exact sums of three bfloat16 values each (split_parts.cuh, gemm_split_f32.cu), six products
// of parts for each; a page's scores are sums of 64 products, and a page's output leaves tensor memory before it is added to
// the rows' running sums, in float32 registers.  Scores, expf and sums are float32 as in attention_tile_f32.cu, and the
// results are closer to 64 bits than there (its chains of multiply-adds are longer).  A row with an infinity or a value that is no number
// among its sums (the parts of an infinity are none, and a weight of zero does not silence such a value) is made again
// from the keys that it sees by chains of multiply-adds.
//
// Warp 0 issues the products; sixteen worker warps hold a row each thread, a quarter of its 64 scores and of its 64
// outputs: they split a page's keys and values into shared memory (two pages), read the scores, share the rows' maxima
// there, write the weights' parts, add the page before's output, and split the keys two pages ahead and the values one, so that
// scores are always made under the softmax of the page before.  The key range may be
// cut into slices whose records the merge kernel of attention_merge.cuh puts together.
// What bounds it: the workers' instructions, 700 a thread and page (3.1 us a page; the products of a page take 1.2 us under
// them), and 6 us of start, first page and end.  9 heads of 64, attention_tile_f32.cu -> here, merges included: prompts of
// 509, 131 and 384 tokens 55 -> 23.6 us, 1,024 88 -> 32, three of 1,024 228 -> 83, 100 18.5 -> 12.0, 17 after 500 46 -> 11.3;
// distance from 64 bits 2.4e-7 -> 1.5e-7 (2-norm).  Keys and values of a page split together one page ahead: 4.5 us a page.
// Every wait is bounded, as in gemm_tcgen05.cu.
#include "attention_merge.cuh"
#include "split_parts.cuh"
#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kSaRows = 128, kSaKeys = 64, kSaD = 64, kSaWorkers = 16;
constexpr int kSaThreads = 32 * (1 + kSaWorkers);
constexpr uint32_t kSaPartQ = kSaRows * 128, kSaPartK = kSaKeys * 128;  // bytes of a part: queries or weights, keys or values
constexpr uint32_t kSaStage = 6 * kSaPartK;                             // K parts, then V parts, of a page
constexpr uint32_t kSaSmem = 6 * kSaPartQ + 2 * kSaStage + 1024;

struct SplitAttnArgs {
    const float* q;
    const float* k_cache;
    const float* v_cache;
    const int4* units;
    const int* seq_first_row;
    const int* seq_start;
    const int* seq_count;
    const int* page_table;
    float* out;
    float* partial;
    int* status;
    int q_stride, table_cols, nq, nkv, window, n_splits;
    float scale;
};

// A row's maximum, sum and sixteen outputs from column c0 on, over keys lo to hi - 1, by chains of multiply-adds.
__device__ __noinline__ void split_row_again(const SplitAttnArgs& g, const int* table, int hk, const float* q, int lo, int hi,
                                             int c0, float& m, float& l, float (&acc)[16]) {
    auto row_of = [&](const float* cache, int t) {
        return cache + (((size_t)table[t / kSaKeys] * g.nkv + hk) * kSaKeys + t % kSaKeys) * kSaD;
    };
    auto score = [&](int t) {
        const float* k = row_of(g.k_cache, t);
        float s = 0.f;
        for (int d = 0; d < kSaD; ++d) s = fmaf(q[d], k[d], s);
        return s * g.scale;
    };
    m = -INFINITY;
    l = 0.f;
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    for (int t = lo; t < hi; ++t) m = fmaxf(m, score(t));
    const float base = m == -INFINITY ? 0.f : m;
    for (int t = lo; t < hi; ++t) {
        const float p = expf(score(t) - base);
        const float* v = row_of(g.v_cache, t) + c0;
        l += p;
        for (int i = 0; i < 16; ++i) acc[i] = fmaf(p, v[i], acc[i]);
    }
}

__device__ __forceinline__ void workers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kSaWorkers) : "memory"); }

__global__ void __launch_bounds__(kSaThreads, 1)
attn_split_f32_kernel(const SplitAttnArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = base;                     // three parts [128][64]
    unsigned char* p_s = base + 3 * kSaPartQ;      // ... of the weights
    unsigned char* kv_s = base + 6 * kSaPartQ;     // two pages
    __shared__ __align__(8) uint64_t k_full[2], v_full[2], s_full[2], p_full, pv_full;
    __shared__ float top_s[2][4][kSaRows], sum_s[4][kSaRows];
    __shared__ int bad_s[kSaRows], stop_s[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 unit_of = g.units[blockIdx.x];  // sequence, first query, slice of the tile's keys, slices of the tile
    const int seq = unit_of.x, q0 = unit_of.y, slice = unit_of.z, slices = unit_of.w, hq = blockIdx.y, hk = hq / (g.nq / g.nkv);
    const int rows = min(kSaRows, g.seq_count[seq] - q0);
    const int pos0 = g.seq_start[seq] + q0, row0 = g.seq_first_row[seq] + q0;
    const int* table = g.page_table + (size_t)seq * g.table_cols;
    const int lo = g.window > 0 ? max(0, pos0 - g.window + 1) : 0, hi = pos0 + rows;  // keys that the tile sees
    const int first_page = lo / kSaKeys, all_pages = (hi - 1) / kSaKeys - first_page + 1;
    const int per = (all_pages + slices - 1) / slices;
    const int p_begin = first_page + slice * per;
    const int pages = max(0, min(first_page + all_pages, p_begin + per) - p_begin);

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&k_full[s], kSaWorkers);
            mbar_init(&v_full[s], kSaWorkers);
            mbar_init(&s_full[s], 1);
        }
        mbar_init(&p_full, kSaWorkers);
        mbar_init(&pv_full, 1);
        abort_flag = 0;
        stop_s[0] = stop_s[1] = 0;
        mbar_fence_init();
    }
    if (threadIdx.x < kSaRows) bad_s[threadIdx.x] = 0;
    if (warp == 0) tmem_alloc(&tmem_base_s, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tmem_o = tmem + 128;  // two pages' scores, a page's output
    pdl_wait();
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = instr_desc(kSaRows, kSaKeys), idesc_o = instr_desc(kSaRows, kSaD) | (1u << 16);
            const uint64_t desc_q = smem_desc_k128(smem_addr(q_s)), desc_p = smem_desc_k128(smem_addr(p_s));
            const uint64_t desc_k = smem_desc_k128(smem_addr(kv_s));
            const uint64_t desc_v = smem_desc_mn128(smem_addr(kv_s) + 3 * kSaPartK);
            bool ok = true;
            auto scores = [&](int j) {
                const int s = j & 1;
                ok = ok && mbar_wait(&k_full[s], (uint32_t)(j >> 1) & 1u) && !abort_flag;
                if (!ok) return;
                tc_fence_after();
                const uint64_t dk = desc_advance(desc_k, (uint32_t)s * kSaStage);
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc_mma(tmem + (uint32_t)s * 64, desc_advance(desc_q, split_part_a(p) * kSaPartQ + k * 32),
                               desc_advance(dk, split_part_b(p) * kSaPartK + k * 32), idesc_s, (p | k) != 0);
                tc_commit(&s_full[s]);
            };
            if (pages > 0) scores(0);
            if (pages > 1) scores(1);
            for (int j = 0; j < pages && ok; ++j) {
                ok = mbar_wait(&v_full[j & 1], (uint32_t)(j >> 1) & 1u) && mbar_wait(&p_full, (uint32_t)j & 1u) && !abort_flag;
                if (!ok) break;
                tc_fence_after();
                const uint64_t dv = desc_advance(desc_v, (uint32_t)(j & 1) * kSaStage);
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)  // (sixteen keys further along the weights' rows, and sixteen rows of V)
                        tc_mma(tmem_o, desc_advance(desc_p, split_part_a(p) * kSaPartQ + k * 32),
                               desc_advance(dv, split_part_b(p) * kSaPartK + k * 2048), idesc_o, (p | k) != 0);
                tc_commit(&pv_full);
                if (j + 2 < pages) scores(j + 2);
            }
            if (!ok) abort_flag = 1;
        }
        __syncwarp();
    } else {
        const int worker = warp - 1, r4 = lane >> 3, unit = lane & 7;
        const int row = (warp & 3) * 32 + lane, cg = worker >> 2;  // this thread's query, its 16 scores and 16 outputs
        const int pos = pos0 + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        // keys and values: four rows of the page a warp, eight floats a lane
        const int kv_row = worker * 4 + r4;
        unsigned char* kv_dst = kv_s + kv_row * 128 + ((unit ^ (kv_row & 7)) << 4);
        unsigned long long kr[4], vr[4];
        auto fetch = [&](const float* cache, int j, unsigned long long (&r)[4]) {
            // (rows past the tile's last key count as zeros, whatever the page holds there)
            if (j < pages && (p_begin + j) * kSaKeys + kv_row < hi) {
                load8(cache + (((size_t)table[p_begin + j] * g.nkv + hk) * kSaKeys + kv_row) * kSaD + unit * 8, r);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) r[e] = 0ull;
            }
        };
        auto keep = [&](int j, int offset, uint64_t* full, unsigned long long (&r)[4]) {
            store_parts(kv_dst + (size_t)(j & 1) * kSaStage + offset, kSaPartK, r);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[j & 1]);
        };
        auto next_keys = [&](int j) {
            keep(j, 0, k_full, kr);
            fetch(g.k_cache, j + 1, kr);
        };
        auto next_values = [&](int j) {
            keep(j, 3 * kSaPartK, v_full, vr);
            fetch(g.v_cache, j + 1, vr);
        };
        fetch(g.k_cache, 0, kr);
        fetch(g.v_cache, 0, vr);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = (i * kSaWorkers + worker) * 4 + r4;
            unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
            if (r < rows) load8(g.q + (size_t)(row0 + r) * g.q_stride + (size_t)hq * kSaD + unit * 8, v);
            store_parts(q_s + r * 128 + ((unit ^ (r & 7)) << 4), kSaPartQ, v);
        }
        if (pages > 0) next_keys(0);
        if (pages > 1) next_keys(1);
        if (pages > 0) next_values(0);
        float m = -INFINITY, l = 0.f, alpha = 0.f, acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        bool ok = true;
        auto add_output = [&](int j) {  // page j's, of the weights relative to the maximum at page j
            ok = mbar_wait(&pv_full, (uint32_t)j & 1u) && ok;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            tc_fence_after();
            uint32_t o[16];
            tmem_load16_issue(tmem_o + lanes + (uint32_t)(cg * 16), o);
            tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = fmaf(acc[i], alpha, __uint_as_float(o[i]));
            tc_fence_before();
        };
        for (int j = 0; j < pages; ++j) {
            // (every worker warp leaves this loop at the same page, as all of them meet in its barrier: what one finds out
            // before the barrier of a page, all read after it, in a place that is written again two barriers on)
            ok = mbar_wait(&s_full[j & 1], (uint32_t)(j >> 1) & 1u) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            uint32_t sr[16];
            tmem_load16_issue(tmem + lanes + (uint32_t)((j & 1) * 64 + cg * 16), sr);
            tmem_load_wait();
            tc_fence_before();
            // (the page's scores are made and read: its keys' place and theirs are free)
            if (j + 2 < pages) next_keys(j + 2);
            float s[16], top = -INFINITY;
            const int t0 = (p_begin + j) * kSaKeys;
            // a page that some query of the tile does not see whole
            const bool edge = t0 + kSaKeys - 1 > pos0 || (g.window > 0 && t0 <= pos0 + kSaRows - 1 - g.window);
#pragma unroll
            for (int i = 0; i < 16; ++i) s[i] = __uint_as_float(sr[i]) * g.scale;
            if (edge) {
                // (one comparison for both ends: a key ahead of the query wraps to a large number)
                const unsigned reach = g.window > 0 ? (unsigned)g.window : 0x7fffffffu;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if ((unsigned)(pos - (t0 + cg * 16 + i)) >= reach) s[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) top = fmaxf(top, s[i]);
            top_s[j & 1][cg][row] = top;
            if (!ok || abort_flag) stop_s[j & 1] = 1;
            workers_meet();
            if (stop_s[j & 1]) {
                ok = false;
                break;
            }
            const float m_new = fmaxf(fmaxf(fmaxf(top_s[j & 1][0][row], top_s[j & 1][1][row]),
                                            fmaxf(top_s[j & 1][2][row], top_s[j & 1][3][row])), m);
            const float from = m_new == -INFINITY ? 0.f : m_new;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                s[i] = expf(s[i] - from);
                sum += s[i];
            }
            if (j > 0) add_output(j - 1);
            alpha = m == -INFINITY ? 0.f : expf(m - from);
            l = fmaf(l, alpha, sum);
            m = m_new;
            // (the page before's output has been read, so its products are through with the weights and with its values)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                unsigned long long w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] = pair_of(s[half * 8 + 2 * e], s[half * 8 + 2 * e + 1]);
                store_parts(p_s + row * 128 + (((cg * 2 + half) ^ (row & 7)) << 4), kSaPartQ, w);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full);
            if (j + 1 < pages) next_values(j + 1);
        }
        if (pages > 0 && ok) add_output(pages - 1);
        if (!ok) abort_flag = 1;
        // the row's sum, and whether any of its values is none
        bool fine = true;
        sum_s[cg][row] = l;
#pragma unroll
        for (int i = 0; i < 16; ++i) fine = fine && isfinite(acc[i]);
        if (!fine || !isfinite(l)) bad_s[row] = 1;
        workers_meet();
        l = sum_s[0][row] + sum_s[1][row] + sum_s[2][row] + sum_s[3][row];
        if (row < rows && !abort_flag) {
            if (bad_s[row]) {
                const int from = max(g.window > 0 ? max(0, pos - g.window + 1) : 0, p_begin * kSaKeys);
                split_row_again(g, table, hk, g.q + (size_t)(row0 + row) * g.q_stride + (size_t)hq * kSaD, from,
                                min(pos + 1, (p_begin + pages) * kSaKeys), cg * 16, m, l, acc);
            }
            const size_t at = (size_t)(row0 + row) * g.nq + hq;
            if (g.n_splits == 1) {
                const float inv = l != 0.f ? 1.0f / l : 0.f;
                float* to = g.out + at * kSaD + cg * 16;
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    store4(to + i, make_float4(acc[i] * inv, acc[i + 1] * inv, acc[i + 2] * inv, acc[i + 3] * inv));
            } else {
                float* rec = g.partial + (at * g.n_splits + slice) * (size_t)(kSaD + 2);
                if (cg == 0) *reinterpret_cast<float2*>(rec) = make_float2(m == -INFINITY ? 0.f : m, l);
                if (cg == 1 && slice == slices - 1)  // (the records that other tiles have and this one has not)
                    for (int z = 1; z < g.n_splits - slice; ++z)
                        *reinterpret_cast<float2*>(rec + z * (kSaD + 2)) = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 16; i += 2)
                    *reinterpret_cast<float2*>(rec + 2 + cg * 16 + i) = make_float2(acc[i], acc[i + 1]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
    if (threadIdx.x == 0 && abort_flag && g.status) atomicExch(g.status, 3);
}

}  // namespace nnis

// float32, pages of 64 keys, head size 64, rows of q that start on 32-byte boundaries.  `units`: int32 [n_units, 4] =
// (sequence of the batch, first of 128 queries among this step's tokens of it, slice of their keys, slices these queries have:
// at most n_splits), every slice of every tile once.  Scratch as nnis_attention_tile_f32.
NNIS_API int nnis_attention_split_f32(const void* q, int q_stride, const void* k_cache, const void* v_cache, const int* units,
                                      int n_units, const int* seq_first_row, const int* seq_start, const int* seq_count,
                                      const int* page_table, int table_cols, void* out, float* partial, int n_tokens, int nq,
                                      int nkv, int d, int page_size, int window, float scale, int n_splits, int* status,
                                      cudaStream_t stream) {
    using namespace nnis;
    if (n_units <= 0 || n_tokens <= 0 || nq <= 0 || nkv <= 0 || nq % nkv || table_cols <= 0 || n_splits <= 0 ||
        window < 0 || !units || (n_splits > 1 && !partial))
        return NNIS_ERR_ARGUMENT;
    if (page_size != kSaKeys || d != kSaD || q_stride % 8 || nq > 65535 || n_splits > 64) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) % 32 || (uintptr_t)out % 16 || (uintptr_t)partial % 8 ||
        (uintptr_t)units % 16)
        return NNIS_ERR_ALIGNMENT;
    SplitAttnArgs g{(const float*)q, (const float*)k_cache, (const float*)v_cache, reinterpret_cast<const int4*>(units),
                    seq_first_row, seq_start, seq_count, page_table, (float*)out, partial, status, q_stride, table_cols, nq,
                    nkv, window, n_splits, scale};
    cudaError_t e = cudaFuncSetAttribute(attn_split_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSaSmem);
    if (e != cudaSuccess) return (int)e;
    e = launch_dependent(attn_split_f32_kernel, dim3(n_units, nq), kSaThreads, kSaSmem, stream, g);
    if (e == cudaSuccess && n_splits > 1)
        e = launch_merge<float>(partial, (float*)out, (size_t)n_tokens * nq, d, n_splits, nullptr, stream);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
