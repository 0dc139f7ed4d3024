// What the tokens of two neighbouring chunks of 64 read in a linear recurrence, on the fifth-generation tensor cores:
//     o_i = carry_i S^T q_i + sum_(j <= i) weigh(i, j, q_i . k_j) v_j
// for up to 128 tokens, up to 256 columns of the values, heads of 64 or 128 keys, S the state before the first of them.  All
// operands are float32 and enter the products as the exact sums of three bfloat16 values each (split_parts.cuh); sums leave
// tensor memory every 64 products of their row and are added in registers, as in gemm_split_f32.cu, and what comes out
// no number is made again by chains of multiply-adds.
//
// A CTA of 17 warps: one issues the products; sixteen split operands, read sums, and hold a token and 32 keys or columns each
// thread.  Shared memory: the queries' parts (128 x 64 twice), which the scores and the state meet and the weights replace,
// and a ring of two blocks for what they meet (128 x 64 keys, or 64 x 128 of the state or the values).
// What bounds it: the way of a block through its loads, the splitting, the fence and the sixteen warps' arrivals, 3,300 cycles (the
// products of a block take 1,536, issued in 2,400), and 8,000 cycles of start and 6,000 of end: one CTA has the SM's shared
// memory, so nothing hides them.  Asking for the next block's values after the hand-over instead of before the fence was slower
// (retention's read 30.2 -> 32.4 us).
#pragma once

#include "split_parts.cuh"
#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kCrTokens = 128, kCrCols = 128, kCrTiles = 2, kCrWorkers = 16;
constexpr int kCrThreads = 32 * (1 + kCrWorkers);
constexpr uint32_t kCrPart = 128 * 128;     // bytes of a part of a block: 128 rows of 64, or 2 x 64 rows of 64
constexpr uint32_t kCrBlock = 3 * kCrPart;
constexpr uint32_t kCrSmem = 4 * kCrBlock + 1024;  // two blocks of queries or weights, two of what they meet
constexpr int kCrMaxBlocks = 2 + 2 * kCrTiles + 2 * kCrTiles;

// Rows of the operands, on 32-byte boundaries: token t of the pair is row t % 64 of its chunk's part.
struct ChunkReadRows {
    const float* q[2];
    const float* k[2];
    const float* v[2];           // from the CTA's first column on
    const float* state;          // likewise, or null: nothing before
    int q_stride, k_stride, v_stride, state_stride;
    int count, dim, cols;        // tokens (at most 128), 64 or 128, columns (a multiple of eight, at most 256)
    float q_scale;
};

struct ChunkReadShared {
    uint64_t full[2], done[kCrMaxBlocks];
    uint32_t tmem;
    float sums[4][kCrTokens];   // the weights' sums, 32 keys each
    float dots[kCrTokens];      // `norm` . q
    volatile int abort_flag;
};

__device__ __forceinline__ void chunk_workers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kCrWorkers) : "memory"); }

// Two neighbouring chunks of a sequence: `at` counts such pairs through the sequences, whose first chunks `first` [n_seqs + 1]
// names.  seq = -1: there are fewer.  Each warp looks through 32 sequences at a time.
struct ChunkPair {
    int seq, chunk;
};
__device__ __forceinline__ ChunkPair find_chunk_pair(const int* first, int n_seqs, int at) {
    const int lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        int c0 = 0, pairs = 0;
        if (s0 + lane < n_seqs) {
            c0 = first[s0 + lane];
            pairs = (first[s0 + lane + 1] - c0 + 1) / 2;
        }
        int to = pairs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, to, o);
            if (lane >= o) to += x;
        }
        const unsigned past = __ballot_sync(0xffffffffu, at < to);
        if (past) {
            const int l = __ffs(past) - 1;
            return {s0 + l, __shfl_sync(0xffffffffu, c0 + 2 * (at - (to - pairs)), l)};
        }
        at -= __shfl_sync(0xffffffffu, to, 31);
    }
    return {-1, 0};
}
__device__ __forceinline__ int chunk_pairs_before(const int* first, int seq) {
    int n = 0;
    for (int s = threadIdx.x & 31; s < seq; s += 32) n += (first[s + 1] - first[s] + 1) / 2;
    return __reduce_add_sync(0xffffffffu, n);
}

// Columns of a CTA that reads: two tiles of 128 split 14 blocks of 128 x 64 where two CTAs split 20, and the fewer of all waves
// of CTAs, one to an SM, is faster (four heads of 256 columns: 120 CTAs 35 us, 240 CTAs 42 us).
inline int chunk_read_cols(long long pairs, int vdim, int sms) {
    const auto cost = [&](int cols, int split) { return (pairs * ((vdim + cols - 1) / cols) + sms - 1) / sms * split; };
    return vdim > kCrCols && cost(2 * kCrCols, 14) < cost(kCrCols, 10) ? 2 * kCrCols : kCrCols;
}

// B of 64 rows x 128 columns as it lies (rows of 128 bytes, two runs of 64 columns 8 KB apart), read MN-major.
__device__ __forceinline__ uint64_t chunk_desc_mn(uint32_t smem_byte_addr) {
    uint64_t desc = smem_desc_mn128(smem_byte_addr);
    return (desc & ~((uint64_t)0x3FFF << 16)) | (uint64_t)(8192 >> 4) << 16;
}

// Every thread of the CTA calls it.  `prepare()` runs on every thread before anything that reads what an earlier kernel
// wrote, and ends in a barrier of the CTA; `weigh(i, j, x)` is asked for j <= i < count alone; `norm` (null: none) is a vector
// whose product with every query is wanted; `finish(i, c, x, sum, dot)` takes eight outputs of a token from column c of the
// CTA's on, the sum of the token's weights, and norm . q.
template <typename Prepare, typename Weigh, typename Carry, typename Finish>
__device__ __forceinline__ void chunk_read_split(const ChunkReadRows& g, const float* norm, ChunkReadShared& sh,
                                                 unsigned char* smem_raw, int* status, Prepare prepare, Weigh weigh,
                                                 Carry carry, Finish finish) {
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = base + 2 * kCrBlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&sh.full[0], kCrWorkers);
        mbar_init(&sh.full[1], kCrWorkers);
        for (int b = 0; b < kCrMaxBlocks; ++b) mbar_init(&sh.done[b], 1);
        sh.abort_flag = 0;
        mbar_fence_init();
    }
    if (threadIdx.x < kCrTokens) sh.dots[threadIdx.x] = 0.f;
    if (warp == 0) tmem_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    prepare();
    // Blocks in order: the scores (nd), the first tile's state, the second's (nd each), the tiles' weights times values (np each)
    const int nd = g.dim / 64, np = (g.count + 63) / 64, tiles = (g.cols + kCrCols - 1) / kCrCols;
    const int tile1 = nd + (g.state ? nd : 0), weights0 = g.state ? tile1 + (tiles - 1) * nd : nd;
    const int blocks = weights0 + tiles * np;
    // their block of queries or weights, and the place of their sums in tensor memory: the second tile's state takes that of
    // the scores, the weights that of the first tile's state, each after every thread has read what was there
    auto place_a = [&](int b) { return (uint32_t)(b < weights0 ? b % nd : (b - weights0) % np); };
    auto place_d = [&](int b) {
        return (uint32_t)(b < nd ? b : b < weights0 ? (b < tile1 ? 2 : 0) + b % nd : 2 + (b - weights0) % np) * 128u;
    };

    if (warp == 0) {
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc(128, 128);
            const uint64_t desc_q = smem_desc_k128(smem_addr(base)), desc_k = smem_desc_k128(smem_addr(ring));
            const uint64_t desc_mn = chunk_desc_mn(smem_addr(ring));
            for (int b = 0; b < blocks; ++b) {
                if (!mbar_wait(&sh.full[b & 1], (uint32_t)(b >> 1) & 1u) || sh.abort_flag) {
                    sh.abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const bool scores = b < nd;
                const uint64_t da = desc_advance(desc_q, place_a(b) * kCrBlock);
                const uint64_t db = desc_advance(scores ? desc_k : desc_mn, (uint32_t)(b & 1) * kCrBlock);
                const uint32_t step = scores ? 32 : 2048, id = scores ? idesc : idesc | (1u << 16), to = tmem + place_d(b);
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc_mma(to, desc_advance(da, split_part_a(p) * kCrPart + k * 32),
                               desc_advance(db, split_part_b(p) * kCrPart + k * step), id, (p | k) != 0);
                tc_commit(&sh.done[b]);
            }
        }
        __syncwarp();
    } else {
        const int worker = warp - 1, r4 = lane >> 3, unit = lane & 7;
        const int row = (warp & 3) * 32 + lane, cg = worker >> 2;  // this thread's token, and its 32 keys or columns of a tile
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        bool ok = true;
        auto wait_done = [&](int b) {
            ok = mbar_wait(&sh.done[b], 0) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
        };
        auto zero = [](unsigned long long (&v)[4]) { v[0] = v[1] = v[2] = v[3] = 0ull; };
        // 128 tokens x 64 places of the keys: two items a thread, one of each chunk
        auto token_rows = [&](const float* const (&rows)[2], int stride, int d0, unsigned long long (&v)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = (i * kCrWorkers + worker) * 4 + r4;
                if (t < g.count) load8(rows[i] + (size_t)(t & 63) * stride + d0 + unit * 8, v[i]);
                else zero(v[i]);
            }
        };
        auto keep_tokens = [&](unsigned char* to, unsigned long long (&v)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = (i * kCrWorkers + worker) * 4 + r4;
                store_parts(to + t * 128 + ((unit ^ (t & 7)) << 4), kCrPart, v[i]);
            }
        };
        // what the queries or weights meet in block b, asked for as soon as the block before has left the registers
        unsigned long long vb[2][4];
        auto load_b = [&](int b) {
            if (b < nd) {
                token_rows(g.k, g.k_stride, b * 64, vb);
                return;
            }
            const bool state = b < weights0;
            const int tile = state ? b >= tile1 : (b - weights0) / np, r0 = (state ? b % nd : (b - weights0) % np) * 64;
            const float* rows = state ? g.state + (size_t)r0 * g.state_stride : r0 ? g.v[1] : g.v[0];
            const int stride = state ? g.state_stride : g.v_stride, there = state ? 64 : g.count - r0;
            // 64 rows x 128 columns: a warp two rows at a time, two items a thread
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (i * kCrWorkers + worker) * 2 + (lane >> 4), c = tile * kCrCols + (lane & 15) * 8;
                if (r < there && c < g.cols) load8(rows + (size_t)r * stride + c, vb[i]);
                else zero(vb[i]);
            }
        };
        auto keep_b_and_hand_over = [&](int b) {
            if (b >= 2) wait_done(b - 2);
            unsigned char* to = ring + (size_t)(b & 1) * kCrBlock;
            if (b < nd) {
                keep_tokens(to, vb);
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = (i * kCrWorkers + worker) * 2 + (lane >> 4), c = lane & 15;
                    store_parts(to + (c >> 3) * 8192 + r * 128 + (((c & 7) ^ (r & 7)) << 4), kCrPart, vb[i]);
                }
            }
            if (b + 1 < blocks) load_b(b + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.full[b & 1]);
        };
        auto add_sums = [&](uint32_t place, float (&x)[32]) {
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                uint32_t t[16];
                tmem_load16_issue(tmem + lanes + place + (uint32_t)(cg * 32 + c), t);
                tmem_load_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) x[c + i] += __uint_as_float(t[i]);
            }
        };
        load_b(0);
#pragma unroll 1
        for (int b = 0; b < nd; ++b) {
            unsigned long long va[2][4];
            token_rows(g.q, g.q_stride, b * 64, va);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float dot = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = halves(va[i][e]);
                    const float x0 = x.x * g.q_scale, x1 = x.y * g.q_scale;
                    va[i][e] = pair_of(x0, x1);
                    if (norm) {
                        dot = fmaf(x0, norm[b * 64 + unit * 8 + 2 * e], dot);
                        dot = fmaf(x1, norm[b * 64 + unit * 8 + 2 * e + 1], dot);
                    }
                }
                if (norm) {
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                    if (unit == 0) sh.dots[(i * kCrWorkers + worker) * 4 + r4] += dot;  // (the same thread for every block)
                }
            }
            keep_tokens(base + (size_t)b * kCrBlock, va);
            keep_b_and_hand_over(b);
        }
        for (int b = nd; b < min(tile1, weights0); ++b) keep_b_and_hand_over(b);
        {
            float w[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) w[i] = 0.f;
            for (int b = 0; b < nd; ++b) {
                wait_done(b);
                add_sums(place_d(b), w);
            }
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                w[i] = cg * 32 + i <= row && row < g.count ? weigh(row, cg * 32 + i, w[i]) : 0.f;
                sum += w[i];
            }
            sh.sums[cg][row] = sum;
            for (int b = tile1; b < weights0; ++b) keep_b_and_hand_over(b);
            wait_done(weights0 - 1);  // the queries are no longer read
            if (cg < 2 || np > 1)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    unsigned long long v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = pair_of(w[u * 8 + 2 * e], w[u * 8 + 2 * e + 1]);
                    store_parts(base + (size_t)(cg >> 1) * kCrBlock + row * 128 + ((((cg & 1) * 4 + u) ^ (row & 7)) << 4),
                                kCrPart, v);
                }
        }
        chunk_workers_meet();  // (the weights' sums)
        float acc[32], sum = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += sh.sums[i][row];
        auto begin_tile = [&](int tile) {
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.f;
            if (!g.state) return;
            for (int d = 0; d < nd; ++d) add_sums((uint32_t)((tile ? 0 : 2) + d) * 128u, acc);
            const float f = carry(row);
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] *= f;
        };
        auto end_tile = [&](int tile) {
            if (!ok || row >= g.count) return;
            const int c0 = tile * kCrCols + cg * 32, there = g.cols - c0;
            bool fine = true;
            float all = sum;
#pragma unroll
            for (int i = 0; i < 32; ++i) fine = fine && isfinite(acc[i]);
            if (!fine) {
                const float* q = (row < 64 ? g.q[0] : g.q[1]) + (size_t)(row & 63) * g.q_stride;
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = 0.f;
                if (g.state) {
#pragma unroll 1
                    for (int d = 0; d < g.dim; ++d) {
                        const float* s = g.state + (size_t)d * g.state_stride + c0;
                        const float x = q[d] * g.q_scale;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < there) acc[i] = fmaf(x, s[i], acc[i]);
                    }
                    const float f = carry(row);
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[i] *= f;
                }
                all = 0.f;
#pragma unroll 1
                for (int j = 0; j <= row; ++j) {
                    const float* k = (j < 64 ? g.k[0] : g.k[1]) + (size_t)(j & 63) * g.k_stride;
                    const float* v = (j < 64 ? g.v[0] : g.v[1]) + (size_t)(j & 63) * g.v_stride + c0;
                    float x = 0.f;
#pragma unroll 1
                    for (int d = 0; d < g.dim; ++d) x = fmaf(q[d] * g.q_scale, k[d], x);
                    x = weigh(row, j, x);
                    all += x;
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (i < there) acc[i] = fmaf(x, v[i], acc[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; i += 8)
                if (i < there) finish(row, c0 + i, acc + i, all, sh.dots[row]);
        };
        begin_tile(0);
        for (int p = 0; p < np; ++p) keep_b_and_hand_over(weights0 + p);
#pragma unroll 1
        for (int tile = 0; tile < tiles; ++tile) {
            const bool more = tile + 1 < tiles;
#pragma unroll 1
            for (int p = 0; p < np; ++p) {
                const int b = weights0 + tile * np + p;
                wait_done(b);
                add_sums(place_d(b), acc);
                if (more) keep_b_and_hand_over(b + np);  // its sums take the place of those just read
            }
            end_tile(tile);
            if (more) begin_tile(tile + 1);
        }
        if (!ok) sh.abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && sh.abort_flag && status) atomicExch(status, 3);
}

// What the same tokens add to the state: sum_t weight_t k_t v_t^T, and to `norm` sum_t weight_t k_t, in the same way: the
// weighed keys of 64 tokens (both operands lie as they are, one row of 128 a token) meet the values, one block of products for
// 64 tokens and 128 columns.  g.q, g.state and g.q_scale are not looked at; `norm` is null but for the first columns;
// `finish(d, c, x)` takes eight sums of a row from column c of the CTA's on.
template <typename Prepare, typename Weight, typename Finish>
__device__ __forceinline__ void chunk_sum_split(const ChunkReadRows& g, float* norm, ChunkReadShared& sh,
                                                unsigned char* smem_raw, int* status, Prepare prepare, Weight weight,
                                                Finish finish) {
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = base + 2 * kCrBlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&sh.full[0], kCrWorkers);
        mbar_init(&sh.full[1], kCrWorkers);
        for (int b = 0; b < kCrMaxBlocks; ++b) mbar_init(&sh.done[b], 1);
        sh.abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    prepare();
    const int np = (g.count + 63) / 64, tiles = (g.cols + kCrCols - 1) / kCrCols, blocks = np * tiles;  // block p * tiles + tile

    if (warp == 0) {
        if (lane == 0) {
            constexpr uint32_t id = instr_desc(128, 128) | (3u << 15);
            const uint64_t desc_k = chunk_desc_mn(smem_addr(base)), desc_v = chunk_desc_mn(smem_addr(ring));
            for (int b = 0; b < blocks; ++b) {
                if (!mbar_wait(&sh.full[b & 1], (uint32_t)(b >> 1) & 1u) || sh.abort_flag) {
                    sh.abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint64_t da = desc_advance(desc_k, (uint32_t)(b / tiles) * kCrBlock);
                const uint64_t db = desc_advance(desc_v, (uint32_t)(b & 1) * kCrBlock);
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc_mma(tmem + b * 128, desc_advance(da, split_part_a(p) * kCrPart + k * 2048),
                               desc_advance(db, split_part_b(p) * kCrPart + k * 2048), id, (p | k) != 0);
                tc_commit(&sh.done[b]);
            }
        }
        __syncwarp();
    } else {
        const int worker = warp - 1, half = lane >> 4, c8 = lane & 15;
        bool ok = true;
        auto wait_done = [&](int b) {
            ok = mbar_wait(&sh.done[b], 0) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
        };
        // 64 tokens x 128 places: a warp two tokens at a time, two items a thread
        auto load = [&](const float* rows, int stride, int there, int c, int cols, unsigned long long (&v)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (i * kCrWorkers + worker) * 2 + half;
                if (r < there && c < cols) load8(rows + (size_t)r * stride + c, v[i]);
                else v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0ull;
            }
        };
        auto keep = [&](unsigned char* to, unsigned long long (&v)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (i * kCrWorkers + worker) * 2 + half;
                store_parts(to + (c8 >> 3) * 8192 + r * 128 + (((c8 & 7) ^ (r & 7)) << 4), kCrPart, v[i]);
            }
        };
        unsigned long long va[2][4], vb[2][4];
        auto load_k = [&](int p) { load(p ? g.k[1] : g.k[0], g.k_stride, g.count - p * 64, c8 * 8, g.dim, va); };
        auto load_v = [&](int b) {
            const int p = b / tiles;
            load(p ? g.v[1] : g.v[0], g.v_stride, g.count - p * 64, b % tiles * kCrCols + c8 * 8, g.cols, vb);
        };
        float ns[8] = {};
        load_k(0);
        load_v(0);
#pragma unroll 1
        for (int b = 0; b < blocks; ++b) {
            if (b % tiles == 0) {
                const int p = b / tiles;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float w = weight(p * 64 + (i * kCrWorkers + worker) * 2 + half);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 x = halves(va[i][e]);
                        va[i][e] = pair_of(x.x * w, x.y * w);
                        ns[2 * e] += x.x * w;
                        ns[2 * e + 1] += x.y * w;
                    }
                }
                keep(base + (size_t)p * kCrBlock, va);
                if (p + 1 < np) load_k(p + 1);
            }
            if (b >= 2) wait_done(b - 2);
            keep(ring + (size_t)(b & 1) * kCrBlock, vb);
            if (b + 1 < blocks) load_v(b + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.full[b & 1]);
        }
        for (int b = max(0, blocks - 2); b < blocks; ++b) wait_done(b);
        if (norm) {  // 32 half-warps' sums, in the place of the weighed keys
            float* part = reinterpret_cast<float*>(base);
#pragma unroll
            for (int e = 0; e < 8; ++e) part[(worker * 2 + half) * 128 + c8 * 8 + e] = ns[e];
            chunk_workers_meet();
            const int d = threadIdx.x - 32;
            if (d < g.dim) {
                float sum = 0.f;
#pragma unroll 8
                for (int i = 0; i < 2 * kCrWorkers; ++i) sum += part[i * 128 + d];
                norm[d] = sum;
            }
        }
        const int row = (warp & 3) * 32 + lane, cg = worker >> 2;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
#pragma unroll 1
        for (int tile = 0; tile < tiles; ++tile) {
            const int c0 = tile * kCrCols + cg * 32, there = g.cols - c0;
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.f;
            for (int p = 0; p < np; ++p) {
#pragma unroll
                for (int c = 0; c < 32; c += 16) {
                    uint32_t t[16];
                    tmem_load16_issue(tmem + lanes + (uint32_t)((p * tiles + tile) * 128 + cg * 32 + c), t);
                    tmem_load_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(t[i]);
                }
            }
            if (!ok || row >= g.dim) continue;
            bool fine = true;
#pragma unroll
            for (int i = 0; i < 32; ++i) fine = fine && isfinite(acc[i]);
            if (!fine) {
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = 0.f;
#pragma unroll 1
                for (int t = 0; t < g.count; ++t) {
                    const float x = (t < 64 ? g.k[0] : g.k[1])[(size_t)(t & 63) * g.k_stride + row] * weight(t);
                    const float* v = (t < 64 ? g.v[0] : g.v[1]) + (size_t)(t & 63) * g.v_stride + c0;
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (i < there) acc[i] = fmaf(x, v[i], acc[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; i += 8)
                if (i < there) finish(row, c0 + i, acc + i);
        }
        if (!ok) sh.abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && sh.abort_flag && status) atomicExch(status, 3);
}

}  // namespace nnis
