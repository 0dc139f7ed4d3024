// Prompt attention on the fifth-generation tensor cores for wide heads: keys of 96, 128 or 192 values, values of 64
// or 128, packed query tokens of several sequences, each over the keys of its own sequence up to its own position
// (and within the window, if there is one).  Two forms of the keys:
//   paged      K and V pages of the cache, query heads in groups (head size 128);
//   expanded   rows of a buffer [R, ...], a sequence's positions one after another from a multiple of 64 on: a head's
//              plain key values and its values side by side, and a part of the key that all heads share in a buffer
//              of its own (latent attention whose latents have been multiplied out for a prompt).
//
// A CTA has one query head and one or two tiles of 128 queries of a sequence, which share the pages of 64 keys that
// come by TMA into rings.  Its roles:
//   warp 0      one lane issues TMA loads: the Q tiles once, then K a page at a time; warp 3 the same for V (rings of
//               their own: a page's K is done with as soon as its scores are, its V a softmax later);
//   warp 1      allocates tensor memory; one lane issues S[128, 64] = Q K^T for either tile (two buffers each);
//   warp 2      one lane issues O[128, DV] += P V for either tile;
//   warps 4-7   softmax of the first tile, warps 8-11 of the second: a thread has one query row, reads its 64 scores
//               from tensor memory, masks them, keeps the row's maximum and sum (float32, exp2) and writes P
//               (bfloat16) into shared memory in the 128-byte-swizzled K-major layout that the second product reads.
// O stays in tensor memory: the maximum that P is taken against is only raised when a page's maximum exceeds it by
// more than 8 (a factor 256, harmless in float32 and bfloat16); then the warp waits for the products so far and
// multiplies its rows of O.  Sum and output are relative to the same maximum, so the result is the exact softmax.
//
// A weight of zero does not take an infinity or a NaN out of a product, and a page holds tokens that a query of its tile
// does not see: later ones, ones that its window has passed, slots that nobody has filled.  So a row whose sum of weights
// is a number but whose output is not is made again by its thread, from what it sees alone (wide_redo_row).  (Taking such
// values out of V before the product, in warp 2 or in warp 0, took 4,096 tokens from 128 to 131 and 155 us.)
//
// Why two tiles: shared memory (Q 96 KB of 208 at 192 key values) leaves one CTA to an SM, and one tile's softmax
// would leave the tensor cores idle while it works on a page (about 1,000 cycles, the products of a page 640 to 830);
// with two, one tile's products run under the other's softmax, and a page fetched serves both.  The host pairs a
// prompt's first tile with its last, the second with the last but one: every pair has the same number of pages.
// What bounds it: the softmax warps' special functions and instructions, two warps to a scheduler, and with few tiles
// the longest CTA.  On a B200, 16 heads of 128 over 4 (paged), before (attention_prefill_mma.cu) and now: one prompt
// of 512 tokens 67 -> 15 us, 2,048 169 -> 38, 4,096 408 -> 126 (549 TFLOP/s), eight of 300 81 -> 20.  Expanded, keys
// of 192: 2,048 and 1,311 tokens 71 us, where attention in the latent's space (attention_latent_mma.cu) took 711.
// With K and V in one ring of pages the same took 86: a page's K waited for the V before it to be done with.
// Every wait is bounded; a wait that runs out raises an abort flag that every role sees, all warps still meet at the
// end and tensor memory is freed.
#include <float.h>

#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kWideRows = 128, kWidePage = 64, kWideThreads = 384;
constexpr uint32_t kWideQ = kWideRows * 128, kWideK = kWidePage * 128;  // bytes of 64 columns of a tile, of a page
constexpr float kWideRaise = 8.0f;  // log2 of how far a page's maximum may exceed the one in use

// V as loaded (64 keys by chunks of 64 values, rows of 128 bytes, 128-byte swizzle) as the MN-major B operand: chunks
// of 64 values lie 8 KB apart (leading byte offset), groups of 8 keys 1,024 bytes (stride byte offset).
__device__ __forceinline__ uint64_t wide_desc_v(uint32_t smem_byte_addr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((smem_byte_addr >> 4) & 0x3FFF);
    desc |= (uint64_t)(kWideK >> 4) << 16;
    desc |= (uint64_t)(1024 >> 4) << 32;
    desc |= (uint64_t)1 << 46;  // descriptor version of sm_100
    desc |= (uint64_t)2 << 61;  // SWIZZLE_128B
    return desc;
}

__device__ __forceinline__ float wide_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float wide_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Wait of a thread that has nothing else to do: it may stay suspended for up to two microseconds per try.  False after
// `limit` tries (a quarter of a second).
__device__ __forceinline__ bool wide_idle(uint64_t* bar, uint32_t parity, uint32_t limit = 1u << 17) {
    const uint32_t addr = smem_addr(bar);
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(2000u)
            : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ bool wide_warp_wait(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}

__device__ __forceinline__ void wide_tmem_store16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void wide_tmem_load16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void wide_add_zeros(uint32_t& sum, uint32_t two) {  // sum += 0 * two
    asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(sum) : "r"(two), "r"(0u));
}

struct WideArgs {
    const int* units;          // [n, 4]: sequence, first query of the first tile, of the second (-1: none), unused
    const int* seq_first_row;
    const int* seq_start;
    const int* seq_count;
    const int* page_table;     // paged keys: [sequences, table_cols]
    const int* key_base;       // expanded keys: a sequence's first row
    int table_cols;
    bf16* out;                 // [n_tokens, nq * DV]
    int nq, nkv, q_head, k_head, v_off, window;
    float scale;
    int* status;
    // the operands as they lie in memory, for a row that is made again: rows of q, of plain keys, of the shared part and of
    // values, and the elements between these
    const bf16 *q, *k, *r, *v;
    int q_row, kv_row;
};

// A row of the output again, keys one by one: columns that hold no number although every value seen is one.  A column with
// an infinity or a NaN among the values seen has what their sum is (weights are positive).  m, l: the row's maximum in use
// (scaled, log2 units) and its sum against it.  Slow, and no row of a model whose values are numbers comes here.
template <int KC, int KLAST, int DV, bool PAGED>
__device__ __noinline__ void wide_redo_row(const WideArgs& p, int seq, int hq, int token, int pos, float m, float l) {
    constexpr int SHARED = PAGED ? 0 : KLAST * 16, OWN = (KC - 1) * 64 + KLAST * 16 - SHARED;  // key values of the head, of all heads
    const int hk = hq / (p.nq / p.nkv), lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    const bf16* q = p.q + (size_t)token * p.q_row + (size_t)hq * p.q_head;
    bf16* out = p.out + ((size_t)token * p.nq + hq) * DV;
    auto row_of = [&](int key) {
        return PAGED ? ((size_t)p.page_table[(size_t)seq * p.table_cols + key / kWidePage] * p.nkv + hk) * kWidePage + key % kWidePage
                     : (size_t)p.key_base[seq] + key;
    };
    const size_t k_off = PAGED ? 0 : (size_t)hq * p.k_head, v_off = p.v_off + (PAGED ? 0 : (size_t)hq * DV);
    for (int c0 = 0; c0 < DV; c0 += 8) {
        uint32_t wrong = 0, nan = 0, up = 0, down = 0;  // a bit a column
        for (int e = 0; e < 8; ++e) wrong |= isfinite(to_float(out[c0 + e])) ? 0u : 1u << e;
        for (int key = pos; key >= lo && (wrong & ~nan); --key) {
            const bf16* v = p.v + row_of(key) * p.kv_row + v_off + c0;
            for (int e = 0; e < 8; ++e) {
                const float x = to_float(v[e]);
                if (isfinite(x)) continue;
                if (x > 0.f) up |= 1u << e;
                else if (x < 0.f) down |= 1u << e;
                else nan |= 1u << e;
            }
        }
        nan |= up & down;
        for (int e = 0; e < 8; ++e)
            if (wrong >> e & 1u && (nan | up | down) >> e & 1u)
                out[c0 + e] = from_float<bf16>(nan >> e & 1u ? __int_as_float(0x7fffffff) : up >> e & 1u ? INFINITY : -INFINITY);
        wrong &= ~(nan | up | down);
        if (!wrong) continue;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int key = lo; key <= pos; ++key) {
            const size_t row = row_of(key);
            const bf16* k = p.k + row * p.kv_row + k_off;
            float score = 0.f;
            for (int i = 0; i < OWN; ++i) score = fmaf(to_float(q[i]), to_float(k[i]), score);
            for (int i = 0; i < SHARED; ++i) score = fmaf(to_float(q[OWN + i]), to_float(p.r[row * 64 + i]), score);
            const float w = to_float(from_float<bf16>(wide_ex2(fmaf(score, p.scale * 1.4426950408889634f, -m))));
            const bf16* v = p.v + row * p.kv_row + v_off + c0;
            for (int e = 0; e < 8; ++e)
                if (wrong >> e & 1u) acc[e] = fmaf(w, to_float(v[e]), acc[e]);
        }
        for (int e = 0; e < 8; ++e)
            if (wrong >> e & 1u) out[c0 + e] = from_float<bf16>(acc[e] / l);
    }
}

// KC: chunks of 64 key values, the last one of which has 16 KLAST; DV: values; PAGED: which form of the keys (with
// expanded keys the last chunk is the shared part).
template <int KC, int KLAST, int DV, bool PAGED, int STAGES>
__global__ void __launch_bounds__(kWideThreads, 1)
attn_wide_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_v,
                    const __grid_constant__ WideArgs p) {
    constexpr int VC = DV / 64;
    constexpr uint32_t kStageK = KC * kWideK, kStageV = VC * kWideK, kTileQ = KC * kWideQ;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = base;                    // 2 tiles x KC x [128, 64]
    unsigned char* p_s = q_s + 2 * kTileQ;        // 2 tiles x [128, 64 keys]
    unsigned char* k_s = p_s + 2 * kWideQ;        // stages x KC x [64, 64]
    unsigned char* v_s = k_s + STAGES * kStageK;  // stages x VC x [64, 64]
    __shared__ __align__(8) uint64_t q_full[2], k_full[STAGES], k_empty[STAGES], v_full[STAGES], v_empty[STAGES];
    __shared__ __align__(8) uint64_t s_full[2][2], s_free[2][2], p_ready[2], p_free[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 unit = reinterpret_cast<const int4*>(p.units)[blockIdx.x];
    const int seq = unit.x, hq = blockIdx.y, hk = hq / (p.nq / p.nkv);
    const int count = p.seq_count[seq], start = p.seq_start[seq], row_base = p.seq_first_row[seq];
    // either tile's pages, first .. last; the walk covers both (a tile takes no part in a page outside its own)
    int q0[2], rows[2], first[2], n_pages[2];
    int walk_first = 1 << 30, walk_last = -1;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        q0[t] = t == 0 ? unit.y : unit.z;
        rows[t] = q0[t] < 0 ? 0 : min(kWideRows, count - q0[t]);
        const int pos0 = start + q0[t];
        first[t] = p.window > 0 && rows[t] > 0 ? max(0, pos0 - p.window + 1) / kWidePage : 0;
        n_pages[t] = rows[t] > 0 ? (pos0 + rows[t] - 1) / kWidePage - first[t] + 1 : 0;
        if (rows[t] > 0) {
            walk_first = min(walk_first, first[t]);
            walk_last = max(walk_last, first[t] + n_pages[t] - 1);
        }
    }
    const int walk = walk_last - walk_first + 1;

    if (threadIdx.x == 64) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_r);
        prefetch_tensormap(&map_v);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&q_full[t], 1);
            for (int b = 0; b < 2; ++b) {
                mbar_init(&s_full[t][b], 1);
                mbar_init(&s_free[t][b], 4);  // one arrival per softmax warp
            }
            mbar_init(&p_ready[t], 4);
            mbar_init(&p_free[t], 1);
        }
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&tmem_base_s, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // S of tile t, buffer b at column 128 t + 64 b; O of tile t at 256 + 128 t
    const uint32_t tmem = tmem_base_s;
    pdl_wait();
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (rows[t] <= 0) continue;
                mbar_expect_tx(&q_full[t], kTileQ);
#pragma unroll
                for (int c = 0; c < KC; ++c)
                    tma_load_2d(q_s + t * kTileQ + c * kWideQ, &map_q, hq * p.q_head + c * 64, row_base + q0[t], &q_full[t]);
            }
            const int* table = PAGED ? p.page_table + (size_t)seq * p.table_cols : nullptr;
            const int key0 = PAGED ? 0 : p.key_base[seq];
            int i = 0;
            for (; i < walk; ++i) {
                const int s = i % STAGES;
                if (i >= STAGES && !wide_idle(&k_empty[s], (uint32_t)(i / STAGES - 1) & 1u)) abort_flag = 1;
                if (abort_flag) break;
                unsigned char* stage = k_s + s * kStageK;
                mbar_expect_tx(&k_full[s], kStageK);
                const int row = PAGED ? (table[walk_first + i] * p.nkv + hk) * kWidePage : key0 + (walk_first + i) * kWidePage;
                if (PAGED) {
#pragma unroll
                    for (int c = 0; c < KC; ++c) tma_load_2d(stage + c * kWideK, &map_k, c * 64, row, &k_full[s]);
                } else {
#pragma unroll
                    for (int c = 0; c + 1 < KC; ++c)
                        tma_load_2d(stage + c * kWideK, &map_k, hq * p.k_head + c * 64, row, &k_full[s]);
                    tma_load_2d(stage + (KC - 1) * kWideK, &map_r, 0, row, &k_full[s]);
                }
            }
            if (abort_flag) {  // no copy may land after the CTA has left
                for (int j = max(0, i - STAGES); j < i; ++j) wide_idle(&k_full[j % STAGES], (uint32_t)(j / STAGES) & 1u);
                for (int t = 0; t < 2; ++t)
                    if (rows[t] > 0) wide_idle(&q_full[t], 0);
            }
        }
    } else if (warp == 3) {
        if (lane == 0) {
            const int* table = PAGED ? p.page_table + (size_t)seq * p.table_cols : nullptr;
            const int key0 = PAGED ? 0 : p.key_base[seq];
            int i = 0;
            for (; i < walk; ++i) {
                const int s = i % STAGES;
                if (i >= STAGES && !wide_idle(&v_empty[s], (uint32_t)(i / STAGES - 1) & 1u)) abort_flag = 1;
                if (abort_flag) break;
                mbar_expect_tx(&v_full[s], kStageV);
                const int row = PAGED ? (table[walk_first + i] * p.nkv + hk) * kWidePage : key0 + (walk_first + i) * kWidePage;
#pragma unroll
                for (int c = 0; c < VC; ++c)
                    tma_load_2d(v_s + s * kStageV + c * kWideK, &map_v, (PAGED ? 0 : p.v_off + hq * DV) + c * 64, row, &v_full[s]);
            }
            if (abort_flag)
                for (int j = max(0, i - STAGES); j < i; ++j) wide_idle(&v_full[j % STAGES], (uint32_t)(j / STAGES) & 1u);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc(kWideRows, kWidePage);
            const uint64_t desc_q0 = smem_desc_k128(smem_addr(q_s)), desc_k0 = smem_desc_k128(smem_addr(k_s));
            bool ok = true;
#pragma unroll
            for (int t = 0; t < 2; ++t)
                if (rows[t] > 0) ok = ok && wide_idle(&q_full[t], 0);
            for (int i = 0; ok && i < walk; ++i) {
                const int s = i % STAGES;
                ok = wide_idle(&k_full[s], (uint32_t)(i / STAGES) & 1u) && !abort_flag;
                const uint64_t desc_k = desc_advance(desc_k0, (uint32_t)s * kStageK);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int j = walk_first + i - first[t], b = j & 1;
                    if (!ok || j < 0 || j >= n_pages[t]) continue;
                    if (j >= 2) ok = wide_idle(&s_free[t][b], (uint32_t)((j >> 1) - 1) & 1u);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < KC; ++c)
#pragma unroll
                        for (int k = 0; k < (c + 1 < KC ? 4 : KLAST); ++k)
                            tc_mma(tmem + t * 128 + b * 64, desc_advance(desc_q0, t * kTileQ + c * kWideQ + k * 32),
                                   desc_advance(desc_k, c * kWideK + k * 32), idesc, (c | k) != 0);
                    tc_commit(&s_full[t][b]);
                }
                if (ok) tc_commit(&k_empty[s]);
            }
            if (!ok) abort_flag = 1;
        }
    } else if (warp == 2) {
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc(kWideRows, DV) | (1u << 16);  // B MN-major
            const uint64_t desc_p0 = smem_desc_k128(smem_addr(p_s));
            const uint64_t desc_v0 = wide_desc_v(smem_addr(v_s));
            bool ok = true;
            for (int i = 0; ok && i < walk; ++i) {
                const int s = i % STAGES;
                ok = wide_idle(&v_full[s], (uint32_t)(i / STAGES) & 1u) && !abort_flag;
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int j = walk_first + i - first[t];
                    if (!ok || j < 0 || j >= n_pages[t]) continue;
                    ok = wide_idle(&p_ready[t], (uint32_t)j & 1u) && !abort_flag;
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t desc_p = desc_advance(desc_p0, t * kWideQ);
                    const uint64_t desc_v = desc_advance(desc_v0, (uint32_t)s * kStageV);
#pragma unroll
                    for (int k = 0; k < kWidePage / 16; ++k)
                        tc_mma(tmem + 256 + t * 128, desc_advance(desc_p, k * 32), desc_advance(desc_v, k * 2048), idesc,
                               (j | k) != 0);
                    tc_commit(&p_free[t]);
                }
                if (ok) tc_commit(&v_empty[s]);
            }
            if (!ok) abort_flag = 1;
        }
    } else if (warp >= 4) {
        const int t = (warp - 4) >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t my_s = tmem + t * 128 + lane_base, my_o = tmem + 256 + t * 128 + lane_base;
        const int my_rows = t ? rows[1] : rows[0], pages = t ? n_pages[1] : n_pages[0], page0 = t ? first[1] : first[0];
        const int tile_pos = start + (t ? q0[1] : q0[0]), pos = tile_pos + row;
        const int lo_row = p.window > 0 ? pos - p.window + 1 : 0;
        // the keys every row of this warp sees whole: no masking on such pages
        const int warp_pos_min = tile_pos + quarter * 32;
        const int warp_lo_max = p.window > 0 ? warp_pos_min + 31 - p.window + 1 : 0;
        const float sc = p.scale * 1.4426950408889634f;
        unsigned char* p_row = p_s + t * kWideQ + row * 128;
        float m_run = -INFINITY, l_run = 0.f;  // maximum in use (scaled, log2 units) and sum against it
        bool ok = true;
        for (int j = 0; j < pages; ++j) {
            const int b = j & 1;
            ok = wide_warp_wait(&s_full[t][b], (uint32_t)(j >> 1) & 1u) && !abort_flag;
            if (!ok) break;
            tc_fence_after();
            uint32_t sa[32], sb[32];
            tmem_load32_issue(my_s + b * 64, sa);
            tmem_load32_issue(my_s + b * 64 + 32, sb);
            tmem_load_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[t][b]);  // this buffer may take the page after next
            const int t0 = (page0 + j) * kWidePage;
            if (t0 + 63 > warp_pos_min || t0 < warp_lo_max) {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    if (t0 + c > pos || t0 + c < lo_row) sa[c] = 0xff800000u;  // -inf
                    if (t0 + 32 + c > pos || t0 + 32 + c < lo_row) sb[c] = 0xff800000u;
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 32; c += 4)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    mx[e] = wide_max3(mx[e], __uint_as_float(sa[c + 2 * e]), __uint_as_float(sa[c + 2 * e + 1]));
                    mx[2 + e] = wide_max3(mx[2 + e], __uint_as_float(sb[c + 2 * e]), __uint_as_float(sb[c + 2 * e + 1]));
                }
            const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc);
            const bool raise = m_run != -INFINITY && m_new > m_run + kWideRaise;
            if (m_run == -INFINITY) m_run = m_new;  // nothing summed yet: this row of O is zero
            const bool rescale = j > 0 && __any_sync(0xffffffffu, raise);
            if (rescale) {
                // every product so far has to be in O before it is rescaled
                ok = wide_warp_wait(&p_free[t], (uint32_t)(j - 1) & 1u);
                if (!ok) break;
                tc_fence_after();
                const float alpha = m_run == -INFINITY ? 1.f : exp2f(m_run - m_new);
#pragma unroll 1
                for (int h = 0; h < DV / 16; ++h) {
                    uint32_t ov[16];
                    wide_tmem_load16(my_o + h * 16, ov);
#pragma unroll
                    for (int c = 0; c < 16; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * alpha);
                    wide_tmem_store16(my_o + h * 16, ov);
                }
                l_run *= alpha;
                m_run = m_new;
            }
            const float neg = m_run == -INFINITY ? 0.f : -m_run;
            float ps[4] = {0.f, 0.f, 0.f, 0.f};
            // weights in place: two bfloat16 a word, the first 16 words of either half
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float a0 = wide_ex2(fmaf(__uint_as_float(sa[2 * c]), sc, neg));
                const float a1 = wide_ex2(fmaf(__uint_as_float(sa[2 * c + 1]), sc, neg));
                ps[c & 3] += a0 + a1;
                const __nv_bfloat162 pk = __floats2bfloat162_rn(a0, a1);
                sa[c] = *reinterpret_cast<const uint32_t*>(&pk);
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float a0 = wide_ex2(fmaf(__uint_as_float(sb[2 * c]), sc, neg));
                const float a1 = wide_ex2(fmaf(__uint_as_float(sb[2 * c + 1]), sc, neg));
                ps[c & 3] += a0 + a1;
                const __nv_bfloat162 pk = __floats2bfloat162_rn(a0, a1);
                sb[c] = *reinterpret_cast<const uint32_t*>(&pk);
            }
            l_run += (ps[0] + ps[1]) + (ps[2] + ps[3]);
            if (j > 0 && !rescale) {  // the product that read P of the page before is over
                ok = wide_warp_wait(&p_free[t], (uint32_t)(j - 1) & 1u);
                if (!ok) break;
            }
            // P row: 8 chunks of 8 keys; chunk c lands at 16-byte slot c ^ (row % 8)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                *reinterpret_cast<uint4*>(p_row + ((c ^ (row & 7)) << 4)) =
                    make_uint4(sa[4 * c], sa[4 * c + 1], sa[4 * c + 2], sa[4 * c + 3]);
                *reinterpret_cast<uint4*>(p_row + (((c + 4) ^ (row & 7)) << 4)) =
                    make_uint4(sb[4 * c], sb[4 * c + 1], sb[4 * c + 2], sb[4 * c + 3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads P through the async proxy
            tc_fence_before();                                            // and a rescaled O through tensor memory
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[t]);
        }
        if (ok && pages > 0) ok = wide_warp_wait(&p_free[t], (uint32_t)(pages - 1) & 1u) && !abort_flag;
        if (!ok) {
            abort_flag = 1;
        } else if (pages > 0) {
            tc_fence_after();
            const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
            uint32_t zero[4] = {0u, 0u, 0u, 0u};  // two bfloat16 each: no numbers once an output is none
            bf16* dst = p.out + (size_t)(row_base + (t ? q0[1] : q0[0]) + row) * p.nq * DV + (size_t)hq * DV;
#pragma unroll 1
            for (int h = 0; h < DV / 32; ++h) {
                uint32_t ov[32];
                tmem_load32(my_o + h * 32, ov);
                if (row < my_rows) {
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 pk = __floats2bfloat162_rn(__uint_as_float(ov[c + 2 * e]) * inv,
                                                                            __uint_as_float(ov[c + 2 * e + 1]) * inv);
                            w[e] = *reinterpret_cast<const uint32_t*>(&pk);
                            wide_add_zeros(zero[e], w[e]);
                        }
                        *reinterpret_cast<uint4*>(dst + h * 32 + c) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            tc_fence_before();
            if (((zero[0] | zero[1] | zero[2] | zero[3]) & 0x7fff7fffu) && isfinite(l_run))
                wide_redo_row<KC, KLAST, DV, PAGED>(p, seq, hq, row_base + (t ? q0[1] : q0[0]) + row, pos, m_run, l_run);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && abort_flag && p.status) atomicExch(p.status, 5);
}

template <int KC, int KLAST, int DV, bool PAGED, int STAGES>
static int launch_wide(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mr, const CUtensorMap& mv,
                       const WideArgs& args, int n_units, int pdl, cudaStream_t stream) {
    constexpr int smem = 2 * KC * kWideQ + 2 * kWideQ + STAGES * (KC + DV / 64) * kWideK + 1024;
    static_assert(smem <= 227 * 1024, "one CTA's shared memory");
    auto kernel = attn_wide_tc_kernel<KC, KLAST, DV, PAGED, STAGES>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_units, args.nq);
    cfg.blockDim = dim3(kWideThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kernel, mq, mk, mr, mv, args);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

}  // namespace nnis

// Paged keys: head size 128 (keys and values), pages of 64.  `units`: int32 [n_units, 4] = (sequence of the batch, first
// query of the first tile within this step's tokens of that sequence, first query of the second or -1, 0).  q:
// [n_tokens, nq * 128] bfloat16 with rows `q_stride` elements apart (a multiple of 8).
NNIS_API int nnis_attention_wide_tc(const void* q, int q_stride, int n_tokens, const void* k_cache, const void* v_cache,
                                    long long cache_rows, const int* units, int n_units, const int* seq_first_row,
                                    const int* seq_start, const int* seq_count, const int* page_table, int table_cols,
                                    void* out, int nq, int nkv, int d, int page_size, int window, float scale,
                                    int* status, int pdl, cudaStream_t stream) {
    using namespace nnis;
    if (n_units <= 0 || n_tokens <= 0 || nq <= 0 || nkv <= 0 || nq % nkv || table_cols <= 0 || window < 0 || !units ||
        cache_rows <= 0 || cache_rows >= (1ll << 31) || q_stride < nq * d || !(scale > 0.f))
        return NNIS_ERR_ARGUMENT;
    if (d != 128 || page_size != kWidePage || nq > 65535 || q_stride % 8) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out | (uintptr_t)units) % 16)
        return NNIS_ERR_ALIGNMENT;
    CUtensorMap mq, mk, mv;
    if (!make_map(&mq, q, n_tokens, nq * d, kWideRows, q_stride) || !make_map(&mk, k_cache, cache_rows, d, kWidePage) ||
        !make_map(&mv, v_cache, cache_rows, d, kWidePage))
        return NNIS_ERR_UNSUPPORTED;
    const WideArgs args = {units, seq_first_row, seq_start, seq_count, page_table, nullptr, table_cols, (bf16*)out,
                           nq, nkv, d, d, 0, window, scale, status, (const bf16*)q, (const bf16*)k_cache, nullptr,
                           (const bf16*)v_cache, q_stride, d};
    return launch_wide<2, 4, 128, true, 3>(mq, mk, mk, mv, args, n_units, pdl, stream);
}

// Expanded keys: q [n_tokens, heads * (dim + rot)], kv [n_rows, heads * (dim + vdim)] (all heads' plain keys, then all
// heads' values), kr [n_rows, 64] (the shared part, zeros beyond rot), bfloat16, packed; `key_base`: every sequence's
// first row, a multiple of 64.  dim, rot, vdim = 128, 64, 128 or 64, 32, 64.
NNIS_API int nnis_attention_wide_tc_expanded(const void* q, int n_tokens, const void* kv, const void* kr,
                                             long long n_rows, const int* units, int n_units, const int* key_base,
                                             const int* seq_first_row, const int* seq_start, const int* seq_count,
                                             void* out, int heads, int dim, int rot, int vdim, int window, float scale,
                                             int* status, int pdl, cudaStream_t stream) {
    using namespace nnis;
    if (n_units <= 0 || n_tokens <= 0 || heads <= 0 || window < 0 || !units || !key_base || n_rows <= 0 ||
        n_rows >= (1ll << 31) || !(scale > 0.f))
        return NNIS_ERR_ARGUMENT;
    const bool large = dim == 128 && rot == 64 && vdim == 128, small = dim == 64 && rot == 32 && vdim == 64;
    if ((!large && !small) || heads > 65535) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)kr | (uintptr_t)out | (uintptr_t)units) % 16) return NNIS_ERR_ALIGNMENT;
    CUtensorMap mq, mk, mr;
    if (!make_map(&mq, q, n_tokens, heads * (dim + rot), kWideRows) ||
        !make_map(&mk, kv, n_rows, heads * (dim + vdim), kWidePage) || !make_map(&mr, kr, n_rows, 64, kWidePage))
        return NNIS_ERR_UNSUPPORTED;
    const WideArgs args = {units, seq_first_row, seq_start, seq_count, nullptr, key_base, 0, (bf16*)out,
                           heads, heads, dim + rot, dim, heads * dim, window, scale, status, (const bf16*)q,
                           (const bf16*)kv, (const bf16*)kr, (const bf16*)kv, heads * (dim + rot), heads * (dim + vdim)};
    return large ? launch_wide<3, 4, 128, false, 2>(mq, mk, mr, mk, args, n_units, pdl, stream)
                 : launch_wide<2, 2, 64, false, 4>(mq, mk, mr, mk, args, n_units, pdl, stream);
}
