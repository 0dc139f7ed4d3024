// The products of a linear recurrence taken a chunk of 64 tokens at a time, all in float32 on the CUDA cores: what a
// chunk adds to the state (U = sum_s k_s v_s^T) and what its tokens read (scores of the chunk's own tokens times the
// values, and the state before the chunk).  Operands lie packed per (chunk, head): keys and queries down their values
// [dim][64] for the products over dim, keys by token [64][dim] for the product over tokens, values [64][vp], vp a
// multiple of four; rows past the chunk's last token are zero.
//
// A thread has 8 x 8 outputs in both kernels, read by 16-byte words that neighbours share, multiplied in pairs; the
// operands come by asynchronous copies two slabs ahead.  Bound by the multiply-add pipe: 96 multiply-adds a thread for
// five words of shared memory where scores and the state's product run together, 64 for four elsewhere.
#pragma once

#include "common.cuh"
#include "fma_pairs.cuh"

namespace nnis {

constexpr int kChunkTokens = 64;

// U tile: 64 rows of dim (from d0) x BV columns (from v0), 128 threads.  `keys` [64][dim], `values` [64][vp], `state`
// [dim][vp].  Shared memory: 64 x (64 + BV) floats.
template <int BV>
__device__ __forceinline__ void chunk_update_tile(const float* __restrict__ keys, const float* __restrict__ values,
                                                  float* __restrict__ state, int dim, int vp, int d0, int v0, float* smem) {
    constexpr int C = kChunkTokens, NC = BV / 64;
    float* ks = smem;           // [64 tokens][64]
    float* vs = smem + C * 64;  // [64 tokens][BV]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
    for (int half = 0; half < 2; ++half) {  // two groups of copies: the first half's products run under the second's
        for (int it = tid; it < 32 * 16; it += 128) {
            const int s = half * 32 + (it >> 4), d = (it & 15) * 4;
            const bool in = d0 + d < dim;
            copy16_or_zero(ks + s * 64 + d, keys + (in ? (size_t)s * dim + d0 + d : 0), in);
        }
        for (int it = tid; it < 32 * (BV / 4); it += 128) {
            const int s = half * 32 + it / (BV / 4), j = (it % (BV / 4)) * 4;
            const bool in = v0 + j < vp;
            copy16_or_zero(vs + s * BV + j, values + (in ? (size_t)s * vp + v0 + j : 0), in);
        }
        copy_commit();
    }
    unsigned long long acc[8][2 * NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        if (half == 0) copy_wait<1>();
        else copy_wait<0>();
        __syncthreads();
#pragma unroll 4
        for (int s = half * 32; s < half * 32 + 32; ++s) {
            const float4 kl = load4(ks + s * 64 + ty * 8), kh = load4(ks + s * 64 + ty * 8 + 4);
            const float k[8] = {kl.x, kl.y, kl.z, kl.w, kh.x, kh.y, kh.z, kh.w};
            ulonglong2 v[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) v[c] = *reinterpret_cast<const ulonglong2*>(vs + s * BV + c * 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long ki = both(k[i]);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    fma2(acc[i][2 * c], ki, v[c].x);
                    fma2(acc[i][2 * c + 1], ki, v[c].y);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int d = d0 + ty * 8 + i;
        if (d >= dim) continue;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int j = v0 + c * 64 + tx * 4;
            const float2 a = halves(acc[i][2 * c]), b = halves(acc[i][2 * c + 1]);
            if (j < vp) store4(state + (size_t)d * vp + j, make_float4(a.x, a.y, b.x, b.y));
        }
    }
}

constexpr int kReadStep = 16, kReadStages = 3, kReadLd = kChunkTokens + 4;
template <int BV>
constexpr int chunk_read_floats() {  // shared memory of chunk_read_tile
    return kReadStages * kReadStep * (2 * kChunkTokens + BV) + kChunkTokens * kReadLd;
}

// Outputs of a chunk's 64 tokens, BV columns from v0, 128 threads: thread (tx, ty) ends with rows 8 ty + i and columns
// 64 c + 4 tx + e in acc.  `queries`, `keys` [dim][64], `state` [dim][vp] (null: nothing before the chunk), `values`
// [64][vp].  `weigh(i, j, x)` turns the score of query i and key j into its weight (0 where j is not seen); `carry(i)`
// multiplies what query i reads of the state before the chunk.
template <int BV, typename Weigh, typename Carry>
__device__ __forceinline__ void chunk_read_tile(const float* __restrict__ queries, const float* __restrict__ keys,
                                                const float* __restrict__ state, const float* __restrict__ values,
                                                int dim, int vp, int v0, int count, float* smem,
                                                unsigned long long (&acc)[8][BV / 32], Weigh weigh, Carry carry) {
    constexpr int C = kChunkTokens, NC = BV / 64, STAGE = kReadStep * (2 * C + BV), VROWS = 32;
    static_assert(VROWS * BV <= STAGE, "a slab of values fits a stage");
    float* ps = smem + kReadStages * STAGE;  // [64 keys][68]: key 4 u + e in row 16 e + u
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, warp = tid >> 5;
    const int nd = dim / kReadStep, nv = (count + VROWS - 1) / VROWS, slabs = nd + nv;
    auto bring = [&](int i) {
        float* st = smem + (i % kReadStages) * STAGE;
        if (i < nd) {
            const int d0 = i * kReadStep;
            for (int it = tid; it < kReadStep * (C / 4); it += 128) {
                copy16_or_zero(st + it * 4, queries + (size_t)d0 * C + it * 4, true);
                copy16_or_zero(st + kReadStep * C + it * 4, keys + (size_t)d0 * C + it * 4, true);
            }
            if (state) {
                for (int it = tid; it < kReadStep * (BV / 4); it += 128) {
                    const int d = it / (BV / 4), j = (it % (BV / 4)) * 4;
                    const bool in = v0 + j < vp;
                    copy16_or_zero(st + 2 * kReadStep * C + it * 4, state + (in ? (size_t)(d0 + d) * vp + v0 + j : 0), in);
                }
            }
        } else if (i < slabs) {
            for (int it = tid; it < VROWS * (BV / 4); it += 128) {
                const int s = (i - nd) * VROWS + it / (BV / 4), j = (it % (BV / 4)) * 4;
                const bool in = v0 + j < vp;
                copy16_or_zero(st + it * 4, values + (in ? (size_t)s * vp + v0 + j : 0), in);
            }
        }
        copy_commit();
    };
    unsigned long long sc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sc[i][0] = sc[i][1] = 0ull;
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;
    }
    bring(0);
    bring(1);
#pragma unroll 1
    for (int i = 0; i < nd; ++i) {
        copy_wait<kReadStages - 2>();
        __syncthreads();  // slab i is there for everyone, and slab i - 1, whose place slab i + 2 takes, is done with
        bring(i + 2);
        const float* st = smem + (i % kReadStages) * STAGE;
        if (state) {
#pragma unroll 4
            for (int d = 0; d < kReadStep; ++d) {
                const float4 ql = load4(st + d * C + ty * 8), qh = load4(st + d * C + ty * 8 + 4);
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(st + (kReadStep + d) * C + tx * 4);
                ulonglong2 s[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    s[c] = *reinterpret_cast<const ulonglong2*>(st + 2 * kReadStep * C + d * BV + c * 64 + tx * 4);
                const float q[8] = {ql.x, ql.y, ql.z, ql.w, qh.x, qh.y, qh.z, qh.w};
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const unsigned long long qr = both(q[r]);
                    fma2(sc[r][0], qr, k.x);
                    fma2(sc[r][1], qr, k.y);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        fma2(acc[r][2 * c], qr, s[c].x);
                        fma2(acc[r][2 * c + 1], qr, s[c].y);
                    }
                }
            }
        } else {
#pragma unroll 4
            for (int d = 0; d < kReadStep; ++d) {
                const float4 ql = load4(st + d * C + ty * 8), qh = load4(st + d * C + ty * 8 + 4);
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(st + (kReadStep + d) * C + tx * 4);
                const float q[8] = {ql.x, ql.y, ql.z, ql.w, qh.x, qh.y, qh.z, qh.w};
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const unsigned long long qr = both(q[r]);
                    fma2(sc[r][0], qr, k.x);
                    fma2(sc[r][1], qr, k.y);
                }
            }
        }
    }
    // weights by key, and the state's part scaled
    {
        float w[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float2 a = halves(sc[r][0]), b = halves(sc[r][1]);
            const int i = ty * 8 + r;
            w[r][0] = weigh(i, tx * 4, a.x);
            w[r][1] = weigh(i, tx * 4 + 1, a.y);
            w[r][2] = weigh(i, tx * 4 + 2, b.x);
            w[r][3] = weigh(i, tx * 4 + 3, b.y);
            const float f = carry(i);
#pragma unroll
            for (int j = 0; j < 2 * NC; ++j) {
                const float2 x = halves(acc[r][j]);
                acc[r][j] = pair_of(x.x * f, x.y * f);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            store4(ps + (e * 16 + tx) * kReadLd + ty * 8, make_float4(w[0][e], w[1][e], w[2][e], w[3][e]));
            store4(ps + (e * 16 + tx) * kReadLd + ty * 8 + 4, make_float4(w[4][e], w[5][e], w[6][e], w[7][e]));
        }
    }
#pragma unroll 1
    for (int i = nd; i < slabs; ++i) {
        copy_wait<kReadStages - 2>();
        __syncthreads();  // (the weights are there too)
        bring(i + 2);
        const float* st = smem + (i % kReadStages) * STAGE;
        // (a warp's queries end at 16 (warp + 1); on its last sixteen keys a value is read only with a weight, as what a
        // later token brings may be no number)
#pragma unroll 1
        for (int u = 0; u < VROWS / 4; ++u) {
            const int key = (i - nd) * VROWS + u * 4;
            if (key >= 16 * (warp + 1)) break;
            const bool edge = key >= 16 * warp;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* pr = ps + (e * 16 + (i - nd) * (VROWS / 4) + u) * kReadLd + ty * 8;
                const float4 pl = load4(pr), ph = load4(pr + 4);
                const float p[8] = {pl.x, pl.y, pl.z, pl.w, ph.x, ph.y, ph.z, ph.w};
                ulonglong2 v[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    v[c] = *reinterpret_cast<const ulonglong2*>(st + (u * 4 + e) * BV + c * 64 + tx * 4);
                if (!edge) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const unsigned long long w = both(p[r]);
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            fma2(acc[r][2 * c], w, v[c].x);
                            fma2(acc[r][2 * c + 1], w, v[c].y);
                        }
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        if (p[r] != 0.f) {
                            const unsigned long long w = both(p[r]);
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                fma2(acc[r][2 * c], w, v[c].x);
                                fma2(acc[r][2 * c + 1], w, v[c].y);
                            }
                        }
                    }
                }
            }
        }
    }
    copy_wait<0>();
}

}  // namespace nnis
