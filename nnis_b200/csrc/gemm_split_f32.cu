// float32 matrix product on the fifth-generation tensor cores: C[M, N] (op)= A[M, K] . W[N, K]^T + bias, every float32
// value taken as the exact sum of three bfloat16 values.
//
// A float32 value x has 24 significant bits.  h = bfloat16(x), m = bfloat16(x - h) and l = bfloat16(x - h - m) hold them
// all (both differences are exact) from 2^-109 on; bfloat16 has float32's range of exponents, so no scaling is needed, but
// below that the last part falls under its smallest number, and what is lost is at most 2^-134 a value.  Of the nine
// products of two such sums the six largest are made (h h, h m, m h, m m, h l, l h); what is left out (m l, l m, l l) is
// 2^-26 of a product and less, where float32 rounds every sum at 2^-24.  The tensor cores cut their running sum off instead
// of rounding it, so no sum stays there for long: 64 columns of K at a time, the small products first, and then the 64
// columns' sum is added in registers, by an ordinary float32 addition.  Against 64-bit sums this is closer than the
// chains of float32 multiply-adds of gemm_simt.cu (figures at the bottom of this comment).
//
// A product that is no number (an infinity among the operands: its h is one and its m is none) is made again from the
// operands by a chain of multiply-adds, so infinities come out as they do there.
//
// One CTA works a tile of 128 x BN (BN 64, 128 or 192), KS CTAs of a cluster share the tile's K and add their sums through
// distributed shared memory, in the order of their ranks (the same bits every time).  Roles:
//   warp 0       allocates tensor memory, brings blocks of A in float32 by TMA and issues tcgen05.mma (kind::f16, 128 x BN x 16, A in
//                tensor memory), 24 for 64 columns of K, into one of two to four accumulators;
//   16 others    split: 16 places of a row of A a thread, whose parts go into tensor memory, and W, 32 bytes a load, one block of K
//                ahead in registers, whose parts go into swizzled shared memory (two blocks of K both); they read the
//                accumulator of two blocks before with tcgen05.ld and add it to their registers (a row and a quarter of the
//                columns a thread); at the end they write the tile, through shared memory, so that whole lines leave.
// Splitting on the way in keeps the weights once in memory, as the decode kernels read them.
//
// What bounds it: shared memory and L1, 128 bytes a cycle.  With A's parts in shared memory too the products read 8 KB every 64 cycles
// (BN = 128) beside 96 KB of parts written and 64 KB loaded for 64 columns of K, 2,750 cycles a block; in tensor memory A is written
// (TMA) and read once as float32, and a block moves 250 KB instead of 350: 2,400 cycles, the products alone 1,536.  Adding
// under the splitting is 3 % faster than before or after it, and costs a tile of 192 columns registers that it has not: that one
// adds after it.  Rows x N x K on a B200, cold L2, A's parts in shared memory -> here: 1,024 x 3,072 x 576 51 -> 35 us (128 tiles of 192
// columns in one wave where 192 of 128 are two), 1,024 x 576 x 1,536 30 -> 25, 1,024 x 576 x 576 19.5 -> 17.4,
// 2,048 x 2,048 x 2,048 127 -> 100 (172 TFLOP/s of float32), 17 x 576 x 576 14.3 -> 12.4; the same bits.  Distance from 64-bit sums
// (2-norm, K = 576 / 1,536 / 5,632): 2.2e-7 / 3.5e-7 / 6.7e-7 by chains of multiply-adds, 0.98e-7 / 1.1e-7 / 1.5e-7 here.
// The gated product also applies silu and multiplies: a pass of 7 us over 1,024 x 3,072 less.
// Level with A's parts in shared memory: tiles of 256 x 128 worked by pairs of CTAs (cta_group::2).  Slower: eight warps that
// split and eight that add.
// Every wait is bounded, as in gemm_tcgen05.cu.
// NNIS: crates/nnis-kernels/src/gemm.rs:16-64 (tiled float32 product on CUDA cores).
#include "split_parts.cuh"
#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kSplitM = 128, kSplitK = 64;
constexpr int kSplitWorkers = 16, kSplitThreads = 32 * (1 + kSplitWorkers);  // warps that split and add, and the one that issues
constexpr int kSplitStages = 2;  // blocks of K in parts
constexpr uint32_t kSplitBlockA = kSplitM * kSplitK * 4;       // two tiles of 128 rows of 32 floats
constexpr uint32_t kSplitLeft = 3 * kSplitK / 2;               // columns of tensor memory that the parts of a block of A take
// Accumulators, and columns of one: a tile of 192 columns has two of 96 a block of K, in a ring of three.
__host__ __device__ constexpr int split_accs(int bn) { return bn == 64 ? 4 : bn == 128 ? 2 : 3; }
__host__ __device__ constexpr int split_acc_cols(int bn) { return bn == 192 ? 96 : bn; }
__host__ __device__ constexpr int split_ahead(int bn) { return bn == 192 ? 2 : 3; }  // blocks of A in float32 on their way
__host__ __device__ constexpr uint32_t split_smem(int bn) { return split_ahead(bn) * kSplitBlockA + kSplitStages * 3u * (uint32_t)bn * 128u; }
struct SplitArgs {
    const float* A;
    const float* W;
    const float* bias;
    float* C;
    int M, N, K, mode;  // 1 store, 2 add, 3 gated: W holds gate rows, then up rows; C [M, N / 2] = silu(gate) up
    int* status;
};

// The element (m, n) by a chain of float32 multiply-adds, for sums that are no numbers.
__device__ __noinline__ float split_again(const float* a, const float* w, int K) {
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
    return s;
}

// Four floats at the same place of the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ float4 peer_load4(const float* p, uint32_t rank) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr(p)), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

template <int BN, int KS>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const SplitArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int kSplitAhead = split_ahead(BN), kAccs = split_accs(BN), kAccCols = split_acc_cols(BN), kHalves = BN / kAccCols;
    constexpr bool kUnder = kHalves == 1;  // sums are added under the splitting of two blocks later; else after that of the next
    constexpr uint32_t kPartW = BN * 128, kStage = 3 * kPartW;
    unsigned char* w_stages = base + kSplitAhead * kSplitBlockA;
    __shared__ __align__(8) uint64_t a_here[kSplitAhead], full_bar[kSplitStages], empty_bar[kSplitStages], acc_full[kAccs], acc_empty[kAccs];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;

    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int slice = KS > 1 ? (int)cluster_rank() : 0;
    const int n0 = (blockIdx.x / KS) * BN, m0 = blockIdx.y * kSplitM;
    const int blocks_all = (g.K + kSplitK - 1) / kSplitK;
    // this slice's run of blocks of K
    const int per = (blocks_all + KS - 1) / KS;
    const int first = min(blocks_all, slice * per), blocks = min(per, blocks_all - first);
    const int inter = g.N >> 1;  // mode 3: columns of the output
    // row of W of the tile's column c, or -1
    auto w_row = [&](int c) {
        if (g.mode != 3) return n0 + c < g.N ? n0 + c : -1;
        const int n = n0 / 2 + c % (BN / 2);
        return n < inter ? (c < BN / 2 ? n : inter + n) : -1;
    };

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_a);
        for (int s = 0; s < kSplitAhead; ++s) mbar_init(&a_here[s], 1);
        for (int s = 0; s < kSplitStages; ++s) {
            mbar_init(&full_bar[s], kSplitWorkers);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < kAccs; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kSplitWorkers / kHalves);
        }
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&tmem_base_s, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0), accs = tmem + kSplitStages * kSplitLeft;

    constexpr int kCols = BN / 4;  // columns of the accumulator to a worker warp
    unsigned long long acc[kCols / 2];  // pairs
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) acc[i] = 0ull;
    if (warp == 0) {
        pdl_wait();
        pdl_launch_dependents();
        auto bring = [&](int kb) {
            if (lane || kb >= blocks) return;
            unsigned char* to = base + (kb % kSplitAhead) * kSplitBlockA;
            mbar_expect_tx(&a_here[kb % kSplitAhead], kSplitBlockA);
            tma_load_2d(to, &map_a, (first + kb) * kSplitK, m0, &a_here[kb % kSplitAhead]);
            tma_load_2d(to + kSplitBlockA / 2, &map_a, (first + kb) * kSplitK + 32, m0, &a_here[kb % kSplitAhead]);
        };
        for (int kb = 0; kb < kSplitAhead; ++kb) bring(kb);
        constexpr uint32_t idesc = instr_desc(kSplitM, kAccCols);
        const uint64_t desc_w = smem_desc_k128(smem_addr(w_stages));
        bool ok = true;
#pragma unroll 1
        for (int kb = 0; kb < blocks && ok; ++kb) {
            const int s = kb % kSplitStages;
            ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], (uint32_t)(kb / kSplitStages) & 1u) && !abort_flag);
            if (!ok) break;
            tc_fence_after();
            bring(kb + kSplitAhead);  // (this block's rows of A are in tensor memory)
            const uint32_t left = tmem + (uint32_t)s * kSplitLeft;
#pragma unroll 1
            for (int half = 0; half < kHalves; ++half) {
                const int at = kb * kHalves + half, b = at % kAccs;
                ok = __all_sync(0xffffffffu, at < kAccs || mbar_wait(&acc_empty[b], (uint32_t)(at / kAccs - 1) & 1u));
                if (!ok) break;
                tc_fence_after();
                const uint32_t to = accs + (uint32_t)b * kAccCols;
                const uint64_t dw = desc_advance(desc_w, (uint32_t)s * kStage + (uint32_t)half * kAccCols * 128);
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int k = 0; k < kSplitK / 16; ++k)
                        warp_mma_ts(to, left + split_part_a(p) * (kSplitK / 2) + k * 8, desc_advance(dw, split_part_b(p) * kPartW + k * 32),
                                    idesc, (p | k) != 0);
                if (half == kHalves - 1) warp_commit(&empty_bar[s]);
                warp_commit(&acc_full[b]);
            }
        }
        if (!ok) abort_flag = 1;
        __syncwarp();
    } else {
        // W: a warp splits four rows at a time, eight floats a lane, BN / 64 such items a thread and block of K; A: a thread
        // has 16 places of a row
        const int worker = warp - 1, r4 = lane >> 3, unit = lane & 7, cg = worker >> 2, row = (warp & 3) * 32 + lane;
        constexpr int kItems = BN / (4 * kSplitWorkers);
        unsigned long long v[kItems][4];
        int rows[kItems];
        uint32_t there = 0;  // bit i: the row of item i exists
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const int at = w_row((i * kSplitWorkers + worker) * 4 + r4);
            rows[i] = max(at, 0);
            if (at >= 0) there |= 1u << i;
            v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0ull;  // (rows beyond N are never loaded and stay zero)
        }
        auto load = [&](int i, int kb, uint32_t wanted) {
            if (wanted & (1u << i)) load8(g.W + ((size_t)rows[i] * g.K + (first + kb) * kSplitK + unit * 8), v[i]);
        };
        int k_left = g.K - first * kSplitK - unit * 8;  // columns from this lane's of the next block on
        // (a warp reads and writes the 32 lanes of tensor memory that its number gives it)
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        // the accumulator that holds this warp's columns of block kb
        auto acc_of = [&](int kb) { return kb * kHalves + (kHalves > 1 ? cg >> 1 : 0); };
        auto ask_sums = [&](int kb, int c, uint32_t (&x)[16]) {
            tmem_load16_issue(accs + lanes + (uint32_t)(acc_of(kb) % kAccs * kAccCols + (kHalves > 1 ? cg & 1 : cg) * kCols + c), x);
        };
        auto add_sums = [&](int c, const uint32_t (&x)[16]) {
            tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                asm("{\n\t.reg .b64 p;\n\tmov.b64 p, {%1, %2};\n\tadd.rn.f32x2 %0, %0, p;\n\t}"
                    : "+l"(acc[c / 2 + i]) : "r"(x[2 * i]), "r"(x[2 * i + 1]));
        };
        auto sums_added = [&](int kb) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc_of(kb) % kAccs]);
        };
        auto add_block = [&](int kb) {
            const int done = acc_of(kb);
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[done % kAccs], (uint32_t)(done / kAccs) & 1u) && !abort_flag)) return false;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < kCols; c += 16) {
                uint32_t sum[16];
                ask_sums(kb, c, sum);
                add_sums(c, sum);
            }
            sums_added(kb);
            return true;
        };
        uint32_t wanted = blocks > 0 && k_left > 0 ? there : 0u;
#pragma unroll
        for (int i = 0; i < kItems; ++i) load(i, 0, wanted);  // (weights depend on no kernel)
        pdl_wait();
        bool ok = true;
        // A block of K: the sums of two blocks before are asked for 16 columns at a time and added under the splitting
        // between, so that a warp waits for tensor memory and for its own splits' way as little as its neighbours leave it.
        for (int kb = 0; kb < blocks; ++kb) {
            const int s = kb % kSplitStages, a = kb % kSplitAhead;
            const bool adds = kUnder && kb >= kSplitStages;
            const uint32_t p_empty = (uint32_t)(kb / kSplitStages - 1) & 1u, p_here = (uint32_t)(kb / kSplitAhead) & 1u;
            const int done = adds ? acc_of(kb - kSplitStages) : 0;
            ok = false;
            for (uint32_t i = 0; i < (1u << 22) && !ok; ++i) {  // (all three polled together)
                ok = mbar_try_wait(&a_here[a], p_here);
                if (kb >= kSplitStages) ok = mbar_try_wait(&empty_bar[s], p_empty) & ok;
                if (adds) ok = mbar_try_wait(&acc_full[done % kAccs], (uint32_t)(done / kAccs) & 1u) & ok;
            }
            ok = __all_sync(0xffffffffu, ok && !abort_flag);
            if (!ok) break;
            tc_fence_after();
            uint32_t sum[16];
            if (adds) ask_sums(kb - kSplitStages, 0, sum);
            {
                const unsigned char* from = base + a * kSplitBlockA + (cg >> 1) * (kSplitBlockA / 2) + row * 128;
#pragma unroll
                for (int c = 0; c < 4; c += 2) {  // (eight places at a time: registers)
                    unsigned long long x[4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(from + ((((cg & 1) * 4 + c + i) ^ (row & 7)) << 4));
                        x[2 * i] = y.x;
                        x[2 * i + 1] = y.y;
                    }
                    uint32_t r[4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) r[e] = p < 2 ? next_part(x[e]) : last_part(x[e]);
                        tmem_store_issue(tmem + lanes + (uint32_t)s * kSplitLeft + p * (kSplitK / 2) + cg * 8 + c * 2, r);
                    }
                }
            }
            if (k_left <= 0) {  // columns beyond K
#pragma unroll
                for (int i = 0; i < kItems; ++i) v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0ull;
            }
            k_left -= kSplitK;
            wanted = kb + 1 < blocks && k_left > 0 ? there : 0u;
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                if (adds) {
                    add_sums(i * 16, sum);
                    if (i + 1 < kItems) ask_sums(kb - kSplitStages, (i + 1) * 16, sum);
                    else sums_added(kb - kSplitStages);
                }
                const int row4 = (i * kSplitWorkers + worker) * 4;
                store_parts(w_stages + (size_t)s * kStage + (row4 + r4) * 128 + ((unit ^ ((row4 & 4) + r4)) << 4), kPartW, v[i]);
                load(i, kb + 1, wanted);
                __syncwarp();  // (rows that do not exist load nothing; tensor memory is for whole warps)
            }
            fence_async_shared();
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[s]);
            if (!kUnder && kb > 0 && !(ok = add_block(kb - 1))) break;
        }
        for (int kb = max(0, blocks - (kUnder ? kSplitStages : 1)); kb < blocks && ok; ++kb) ok = add_block(kb);
        if (!ok) abort_flag = 1;
    }

    // ---- the tile: through shared memory, its lines whole ------------------------------------------------------
    // (all products have been read out: the stages are free)
    constexpr int kRow = BN + 4;  // floats between rows: 16-byte stores of neighbouring rows meet no bank twice
    float* sums = reinterpret_cast<float*>(base);
    __syncthreads();
    const int quarter = warp & 3, c0 = warp > 0 ? ((warp - 1) >> 2) * kCols : 0;
    if (warp > 0) {
        float* mine = sums + (quarter * 32 + lane) * kRow + c0;
#pragma unroll
        for (int i = 0; i < kCols; i += 4)
            *reinterpret_cast<ulonglong2*>(mine + i) = make_ulonglong2(acc[i / 2], acc[i / 2 + 1]);
    }
    if constexpr (KS > 1) cluster_meet();
    else __syncthreads();
    if (warp > 0 && !abort_flag) {
        const bool gated = g.mode == 3;
        // a warp's columns of the output, its lanes to a row, four floats each, and the rows it writes at a time
        const int width = gated ? kCols / 2 : kCols, lanes = width / 4, rows_at = 32 / lanes;
        const int out_cols = gated ? inter : g.N;
        const bool by_four = (out_cols & 3) == 0 && (reinterpret_cast<uintptr_t>(g.C) & 15) == 0;
        const int c = ((warp - 1) >> 2) * width + (lane % lanes) * 4, n = (gated ? n0 / 2 : n0) + c;
        constexpr int kSliceRows = (32 / KS + 7) / 8 * 8;  // of the warp's 32: each slice finishes its share
        const int r_end = min(32, (slice + 1) * kSliceRows);
        auto sum_of = [&](const float* at) {
            float4 v = *reinterpret_cast<const float4*>(at);
            if constexpr (KS > 1) {
                v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int z = 0; z < KS; ++z) {
                    const float4 x = peer_load4(at, (uint32_t)z);
                    v = make_float4(v.x + x.x, v.y + x.y, v.z + x.z, v.w + x.w);
                }
            }
            return v;
        };
#pragma unroll 2
        for (int r = slice * kSliceRows; r < r_end; r += rows_at) {
            const int row = quarter * 32 + r + lane / lanes, m = m0 + row;
            if (lane / lanes >= rows_at || r + lane / lanes >= r_end || m >= g.M || n >= out_cols) continue;
            const float* at = sums + row * kRow + c;
            const float4 v = sum_of(at);
            float f[4] = {v.x, v.y, v.z, v.w}, u[4] = {0.f, 0.f, 0.f, 0.f};
            if (gated) {
                const float4 w = sum_of(at + BN / 2);
                u[0] = w.x;
                u[1] = w.y;
                u[2] = w.z;
                u[3] = w.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (n + e >= out_cols) continue;
                if (!isfinite(f[e])) f[e] = split_again(g.A + (size_t)m * g.K, g.W + (size_t)(n + e) * g.K, g.K);
                if (g.bias) f[e] += g.bias[n + e];
                if (gated) {
                    if (!isfinite(u[e])) u[e] = split_again(g.A + (size_t)m * g.K, g.W + (size_t)(inter + n + e) * g.K, g.K);
                    if (g.bias) u[e] += g.bias[inter + n + e];
                    f[e] = f[e] / (1.0f + expf(-f[e])) * u[e];
                }
            }
            float* out = g.C + (size_t)m * out_cols + n;
            if (by_four) {
                float4 o = make_float4(f[0], f[1], f[2], f[3]);
                if (g.mode == 2) {
                    const float4 old = load4(out);
                    o = make_float4(old.x + o.x, old.y + o.y, old.z + o.z, old.w + o.w);
                }
                store4(out, o);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < out_cols) out[e] = g.mode == 2 ? out[e] + f[e] : f[e];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (KS > 1) cluster_meet();  // no CTA leaves while another reads its sums
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && abort_flag && g.status) atomicExch(g.status, 3);
}

template <int BN, int KS>
static int launch_split(const SplitArgs& g, cudaStream_t stream) {
    auto kernel = gemm_split_kernel<BN, KS>;
    constexpr size_t sums = (size_t)kSplitM * (BN + 4) * 4, stages = split_smem(BN);
    constexpr size_t smem = (sums > stages ? sums : stages) + 1024;
    static_assert(smem <= 227 * 1024 - 2048, "one CTA's shared memory");
    CUtensorMap map_a;
    if (!make_map(&map_a, g.A, g.M, g.K, kSplitM, 0, 4)) return NNIS_ERR_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.N + BN - 1) / BN * KS), (unsigned)((g.M + kSplitM - 1) / kSplitM));
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (KS > 1) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs].val.clusterDim.x = KS;
        attr[attrs].val.clusterDim.y = 1;
        attr[attrs++].val.clusterDim.z = 1;
    }
    if (dependent_launches()) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    e = cudaLaunchKernelEx(&cfg, kernel, map_a, g);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

// Width of the tiles and CTAs that share a tile's K: the least cycles by waves of CTAs, a wave's cost as measured (start and
// end 6,000 cycles, 1,500 more for the widest tile or a cluster's meeting; a block of K 2,600, 1,600 and 1,150 at widths 192, 128
// and 64 relative to those).  us at widths x CTAs 64x1, 64x2, 64x4, 128x1, 128x2, 128x4, 192x1: 1,024 x 576 x 1,536 36, 26, 43, 45,
// 32, 37, 67; 1,024 x 3,072 x 576 47, 71, 121, 43, 47, 78, 35; 2,048 x 2,048 x 2,048 147, 154, 222, 101, 117, 148, 141; 256 x 2,048
// x 2,048 41, 28, 35, 50, 33, 25, 75; 500 x 576 x 1,536 34, 24, 31 (144 CTAs), 45, 30, 22, 67.
static int split_shape(int M, int N, int K, int sms) {
    const long m_tiles = (M + kSplitM - 1) / kSplitM;
    const int blocks = (K + kSplitK - 1) / kSplitK;
    long best = -1;
    int shape = 21;
    for (int bn = 192; bn >= 64; bn -= 64)
        for (int ks = 1; ks <= (bn == 192 ? 1 : 4); ks *= 2) {
            if (ks > 1 && blocks < 2 * ks) continue;
            const long resident = ks == 4 ? sms - sms / 9 : sms;  // (of 148 SMs clusters of four fill 132 at a time)
            const long ctas = m_tiles * ((N + bn - 1) / bn) * ks, waves = (ctas + resident - 1) / resident;
            const long cost = waves * (6000 + (ks > 1 || bn == 192 ? 1500 : 0) + (long)((blocks + ks - 1) / ks) * (bn == 192 ? 2600 : bn == 128 ? 1600 : 1150));
            if (best < 0 || cost < best) {
                best = cost;
                shape = bn / 64 * 10 + ks;
            }
        }
    return shape;
}

}  // namespace nnis

// Modes: 1 store, 2 add into C, 3 gated (W = [gate rows; up rows], C [M, N / 2] = silu(gate) up).  `shape` 0: by the rule; else
// (BN / 64) * 10 + KS.  Refuses (NNIS_ERR_UNSUPPORTED) K not a multiple of 8; A and W start on 32-byte
// boundaries.
NNIS_API int nnis_gemm_split_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                                 int mode, int shape, int sm_count, int* status, cudaStream_t stream) {
    using namespace nnis;
    if (M <= 0 || N <= 0 || K <= 0 || !A || !W || !C || mode < 1 || mode > 3) return NNIS_ERR_ARGUMENT;
    if (K % 8 || (mode == 3 && N % 2) || (M + kSplitM - 1) / kSplitM > 65535) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)A | (uintptr_t)W) % 32 || (uintptr_t)C % 4) return NNIS_ERR_ALIGNMENT;
    SplitArgs g{A, W, bias, C, M, N, K, mode, status};
    if (!shape) shape = split_shape(M, N, K, sm_count > 0 ? sm_count : 148);
    switch (shape) {
        case 31: return launch_split<192, 1>(g, stream);
        case 21: return launch_split<128, 1>(g, stream);
        case 22: return launch_split<128, 2>(g, stream);
        case 24: return launch_split<128, 4>(g, stream);
        case 11: return launch_split<64, 1>(g, stream);
        case 12: return launch_split<64, 2>(g, stream);
        case 14: return launch_split<64, 4>(g, stream);
        default: return NNIS_ERR_ARGUMENT;
    }
}
