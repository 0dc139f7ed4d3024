// Retention: linear attention with a fixed decay per head, no softmax and no
// denominator.  Per head, with q and k rotated by position and k scaled by
// dim^-1/2:   S_t = g S_{t-1} + k_t v_t^T,   o_t = S_t^T q_t.
// The state S [dim, vdim] lives in float32 in a per-sequence state area and is
// carried from step to step; everything between the projections and the output
// (angles, rotation, decay, state, the head's unit norm, the gate) is float32.
//
//   retention_scan   a CTA per (sequence, head, 32 columns of vdim) walks the step's
//                    tokens of that sequence in order; warp w holds rows w, w+8, ...
//                    of the state tile in registers.  Steps of single tokens, and key
//                    sizes that the others do not take.
//   retention_in_order   prompts and later portions of them, key sizes 32, 64, 128 and 256:
//                    chunks of 32 tokens in order.  Short ones.
//   retention_pack, retention_update, retention_carry, retention_read   long ones: chunks of
//                    64 tokens side by side, see below.
//   retention_gate   o / rms(o) per head, times silu(g) (or sigmoid(g)), rounded once;
//   retention_gate_joined   the same with one norm over a token's joined heads and a weight per value.
//
// `act` passes q, k and v through silu as they are read; `k_scale` multiplies k (dim^-1/2 in
// retention proper, 1 for a recurrence without a scale).
//
// Packed input rows: [q (H dim) | k (H dim) | v (H vdim) | g (H vdim)].
#include "async_copy.cuh"
#include "chunk_read_split.cuh"
#include "common.cuh"
#include "linear_chunks.cuh"
#include "row_quads.cuh"

namespace nnis {

// a projection's value as it enters the recurrence: as it is, or through silu (`act`)
template <typename T> __device__ __forceinline__ float pre(T x, int act) {
    const float f = to_float(x);
    return act ? f / (1.0f + expf(-f)) : f;
}

template <typename T, int R>
__global__ void __launch_bounds__(256)
retention_scan_kernel(const T* __restrict__ qkvg, const float* __restrict__ freq,
                      const float* __restrict__ decay, float* __restrict__ state,
                      const int* __restrict__ token_pos, const int* __restrict__ token_seq,
                      const int* __restrict__ seq_slots, const int* __restrict__ seq_first_row,
                      const int* __restrict__ seq_start, const int* __restrict__ seq_count,
                      float* __restrict__ o_raw, int heads, int dim, int vdim, int rot_dims, int act, float k_scale) {
    extern __shared__ float smem[];
    pdl_wait();
    pdl_launch_dependents();
    float* qs = smem;             // [dim]
    float* ks = smem + dim;       // [dim]
    float* red = smem + 2 * dim;  // [8][32]
    int unit = blockIdx.x, h = blockIdx.y, col = blockIdx.z * 32 + (threadIdx.x & 31);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int first, start, count, slot;
    if (seq_first_row) {
        first = seq_first_row[unit];
        start = seq_start[unit];
        count = seq_count[unit];
        slot = seq_slots[unit];
    } else {  // one token per row; a row without a sequence has position -1
        first = unit;
        start = token_pos[unit];
        count = start < 0 ? 0 : 1;
        slot = seq_slots[token_seq[unit]];
    }
    if (count <= 0) return;
    const bool live = col < vdim;
    const float g = decay[h];
    float* S = state + (((size_t)slot * heads + h) * dim) * vdim;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int i = warp + 8 * r;
        s[r] = (live && i < dim) ? S[(size_t)i * vdim + col] : 0.f;
    }
    const size_t row_len = (size_t)2 * heads * dim + (size_t)2 * heads * vdim;
    const int half = rot_dims >> 1;
    for (int t = 0; t < count; ++t) {
        const T* row = qkvg + (size_t)(first + t) * row_len;
        const T* qh = row + (size_t)h * dim;
        const T* kh = row + (size_t)heads * dim + (size_t)h * dim;
        float pos = (float)(start + t);
        for (int j = threadIdx.x; j < dim - half; j += 256) {
            if (j < half) {
                float ang = pos * freq[j];
                float c = cosf(ang), sn = sinf(ang);
                float u = pre(qh[j], act), v = pre(qh[j + half], act);
                qs[j] = u * c - v * sn;
                qs[j + half] = v * c + u * sn;
                u = pre(kh[j], act);
                v = pre(kh[j + half], act);
                ks[j] = (u * c - v * sn) * k_scale;
                ks[j + half] = (v * c + u * sn) * k_scale;
            } else {
                qs[j + half] = pre(qh[j + half], act);
                ks[j + half] = pre(kh[j + half], act) * k_scale;
            }
        }
        __syncthreads();
        float v = live ? pre(row[(size_t)2 * heads * dim + (size_t)h * vdim + col], act) : 0.f;
        float o = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            int i = warp + 8 * r;
            if (i < dim) {
                s[r] = fmaf(g, s[r], ks[i] * v);
                o = fmaf(s[r], qs[i], o);
            }
        }
        red[warp * 32 + lane] = o;
        __syncthreads();
        if (warp == 0 && live) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += red[w * 32 + lane];
            o_raw[((size_t)(first + t) * heads + h) * vdim + col] = sum;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int i = warp + 8 * r;
        if (live && i < dim) S[(size_t)i * vdim + col] = s[r];
    }
}

// Short prompts: chunks of 32 tokens in order, one kernel.  A CTA owns (sequence, head, 32 columns of vdim) and walks the
// chunks with its tile of S in shared memory; q and k of the chunk are rotated once into shared memory.  Within a chunk of
// C tokens, with A[i][j] = (q_i . k_j) g^(i-j) for j <= i and S the state before it:
//     o_i = sum_j A[i][j] v_j + g^(i+1) S^T q_i        S <- g^C S + sum_j g^(C-1-j) k_j v_j^T
constexpr int kRetChunk = 32;

// DR4: dim / 32 (the kernel takes dim = 32, 64, 128, 256; a warp owns dim / 8 rows of the
// state in the update).  The three products are tiled in registers: 2 x 2 entries of A per
// thread, four rows of the output per thread, dim / 8 rows of the state per thread, with
// q and k read as float4 along dim.
template <typename T, int DR4>
__global__ void __launch_bounds__(256)
retention_in_order_kernel(const T* __restrict__ qkvg, const float* __restrict__ freq,
                       const float* __restrict__ decay, float* __restrict__ state,
                       const int* __restrict__ seq_slots, const int* __restrict__ seq_first_row,
                       const int* __restrict__ seq_start, const int* __restrict__ seq_count,
                       float* __restrict__ o_raw, int heads, int vdim, int rot_dims, int act, float k_scale) {
    constexpr int C = kRetChunk, dim = 32 * DR4, ld = dim + 4, DR = 4 * DR4;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                  // [C][dim + 4]
    float* ks = qs + C * ld;           // [C][dim + 4]
    float* Ss = ks + C * ld;           // [dim][32]
    float* As = Ss + dim * 32;         // [C][C + 1]
    float* vs = As + C * (C + 1);      // [C][32]
    float* pw = vs + C * 32;           // [C + 1]: g^n
    const int h = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    const int col = blockIdx.z * 32 + lane;
    const int unit = blockIdx.x, first = seq_first_row[unit], start = seq_start[unit], count = seq_count[unit];
    if (count <= 0) return;
    const bool live = col < vdim;
    const float g = decay[h];
    float* S = state + (((size_t)seq_slots[unit] * heads + h) * dim) * vdim;
    for (int d = warp; d < dim; d += 8) Ss[d * 32 + lane] = live ? S[(size_t)d * vdim + col] : 0.f;
    for (int it = tid; it < 2 * C * ld; it += 256) qs[it] = 0.f;  // (rows beyond a short chunk)
    if (tid == 0) {
        float p = 1.f;
        for (int n = 0; n <= C; ++n) {
            pw[n] = p;
            p *= g;
        }
    }
    const size_t row_len = (size_t)2 * heads * dim + (size_t)2 * heads * vdim;
    const int half = rot_dims >> 1, per_tok = dim - half;
    for (int t0 = 0; t0 < count; t0 += C) {
        const int cnt = min(C, count - t0);
        __syncthreads();  // the chunk before is done with qs, ks, vs, As; Ss is up to date
        for (int it = tid; it < cnt * per_tok; it += 256) {
            int i = it / per_tok, j = it - i * per_tok;
            const T* row = qkvg + (size_t)(first + t0 + i) * row_len;
            const T* qh = row + (size_t)h * dim;
            const T* kh = row + (size_t)heads * dim + (size_t)h * dim;
            if (j < half) {
                float ang = (float)(start + t0 + i) * freq[j];
                float c = cosf(ang), sn = sinf(ang);
                float u = pre(qh[j], act), v = pre(qh[j + half], act);
                qs[i * ld + j] = u * c - v * sn;
                qs[i * ld + j + half] = v * c + u * sn;
                u = pre(kh[j], act);
                v = pre(kh[j + half], act);
                ks[i * ld + j] = (u * c - v * sn) * k_scale;
                ks[i * ld + j + half] = (v * c + u * sn) * k_scale;
            } else {
                qs[i * ld + j + half] = pre(qh[j + half], act);
                ks[i * ld + j + half] = pre(kh[j + half], act) * k_scale;
            }
        }
        for (int it = tid; it < C * 32; it += 256) {
            int i = it >> 5;
            float v = 0.f;
            if (i < cnt && live)
                v = pre(qkvg[(size_t)(first + t0 + i) * row_len + (size_t)2 * heads * dim +
                             (size_t)h * vdim + col], act);
            vs[it] = v;
        }
        __syncthreads();
        {   // A[i][j] = (q_i . k_j) g^(i - j) for j <= i: a 2 x 2 tile per thread
            const int i0 = (tid >> 4) * 2, j0 = (tid & 15) * 2;
            float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f;
            if (j0 <= i0 + 1) {
                const float4* q0 = reinterpret_cast<const float4*>(qs + i0 * ld);
                const float4* q1 = reinterpret_cast<const float4*>(qs + (i0 + 1) * ld);
                const float4* k0 = reinterpret_cast<const float4*>(ks + j0 * ld);
                const float4* k1 = reinterpret_cast<const float4*>(ks + (j0 + 1) * ld);
#pragma unroll 4
                for (int d = 0; d < dim / 4; ++d) {
                    float4 x0 = q0[d], x1 = q1[d], y0 = k0[d], y1 = k1[d];
                    a00 = fmaf(x0.x, y0.x, fmaf(x0.y, y0.y, fmaf(x0.z, y0.z, fmaf(x0.w, y0.w, a00))));
                    a01 = fmaf(x0.x, y1.x, fmaf(x0.y, y1.y, fmaf(x0.z, y1.z, fmaf(x0.w, y1.w, a01))));
                    a10 = fmaf(x1.x, y0.x, fmaf(x1.y, y0.y, fmaf(x1.z, y0.z, fmaf(x1.w, y0.w, a10))));
                    a11 = fmaf(x1.x, y1.x, fmaf(x1.y, y1.y, fmaf(x1.z, y1.z, fmaf(x1.w, y1.w, a11))));
                }
            }
            As[i0 * (C + 1) + j0] = j0 <= i0 ? a00 * pw[i0 - j0] : 0.f;
            As[i0 * (C + 1) + j0 + 1] = j0 + 1 <= i0 ? a01 * pw[i0 - j0 - 1] : 0.f;
            As[(i0 + 1) * (C + 1) + j0] = j0 <= i0 + 1 ? a10 * pw[i0 + 1 - j0] : 0.f;
            As[(i0 + 1) * (C + 1) + j0 + 1] = j0 <= i0 ? a11 * pw[i0 - j0] : 0.f;
        }
        __syncthreads();
        {   // outputs: rows 4 warp .. 4 warp + 3, column = lane
            const int i0 = warp * 4;
            float inter[4] = {0.f, 0.f, 0.f, 0.f}, intra[4] = {0.f, 0.f, 0.f, 0.f};
            if (i0 < cnt) {
#pragma unroll 2
                for (int d = 0; d < dim; d += 4) {
                    float s0 = Ss[d * 32 + lane], s1 = Ss[(d + 1) * 32 + lane];
                    float s2 = Ss[(d + 2) * 32 + lane], s3 = Ss[(d + 3) * 32 + lane];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        float4 x = *reinterpret_cast<const float4*>(qs + (i0 + r) * ld + d);
                        inter[r] = fmaf(x.x, s0, fmaf(x.y, s1, fmaf(x.z, s2, fmaf(x.w, s3, inter[r]))));
                    }
                }
                for (int j = 0; j < i0; ++j) {
                    float v = vs[j * 32 + lane];
#pragma unroll
                    for (int r = 0; r < 4; ++r) intra[r] = fmaf(As[(i0 + r) * (C + 1) + j], v, intra[r]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {  // (what a later token brings may be no number)
                    float v = vs[(i0 + j) * 32 + lane];
#pragma unroll
                    for (int r = j; r < 4; ++r) intra[r] = fmaf(As[(i0 + r) * (C + 1) + i0 + j], v, intra[r]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (live && i0 + r < cnt)
                        o_raw[((size_t)(first + t0 + i0 + r) * heads + h) * vdim + col] =
                            fmaf(pw[i0 + r + 1], inter[r], intra[r]);
            }
        }
        __syncthreads();
        {   // the state after the chunk: rows warp * DR .. + DR - 1, column = lane
            const int d0 = warp * DR;
            float acc[DR];
#pragma unroll
            for (int r = 0; r < DR; ++r) acc[r] = 0.f;
            for (int j = 0; j < cnt; ++j) {
                float v = pw[cnt - 1 - j] * vs[j * 32 + lane];
#pragma unroll
                for (int r4 = 0; r4 < DR4; ++r4) {
                    float4 k = *reinterpret_cast<const float4*>(ks + j * ld + d0 + 4 * r4);
                    acc[4 * r4] = fmaf(k.x, v, acc[4 * r4]);
                    acc[4 * r4 + 1] = fmaf(k.y, v, acc[4 * r4 + 1]);
                    acc[4 * r4 + 2] = fmaf(k.z, v, acc[4 * r4 + 2]);
                    acc[4 * r4 + 3] = fmaf(k.w, v, acc[4 * r4 + 3]);
                }
            }
#pragma unroll
            for (int r = 0; r < DR; ++r) Ss[(d0 + r) * 32 + lane] = fmaf(pw[cnt], Ss[(d0 + r) * 32 + lane], acc[r]);
        }
    }
    __syncthreads();
    for (int d = warp; d < dim; d += 8)
        if (live) S[(size_t)d * vdim + col] = Ss[d * 32 + lane];
}

// Longer prompts: the same a chunk of 64 tokens at a time, chunks side by side, all in float32.  Four kernels: `pack` turns q, k and v of every (chunk, head) into the layouts that
// the products read (rotated once, not once per tile of columns); `update` makes what every chunk adds to the state, all
// chunks side by side; `carry` walks a sequence's chunks in order and leaves the state before each of them, and the
// slot's state; `read` makes the outputs, all chunks side by side.  The products are linear_chunks.cuh's.  More chunks
// than the scratch holds go through the four kernels in waves, the slot's state from one to the next (the same bits: the
// state is float32 there too).
// Before, chunks of 32 in runs of 256 tokens from zero, 32 columns a CTA with A made again for each, 2 x 2 entries of A
// and 4 x 1 of the output a thread, took 495 us for 2,048 tokens and 8 heads of 128 x 256 on a B200 (chunk 351, prefix
// 30, carry 114); these kernels 143 (pack 37, update 25, carry 12, read 66: 22 TFLOP/s of multiply-adds on the CUDA cores).
// Keys of 64 and 128 have `update` and `read` on the tensor cores, by pairs of chunks (below): 70.

// A packed (chunk, head): queries [dim][64], keys [dim][64], keys times g^(C-1-j) [64][dim], values [64][vp].
__host__ __device__ __forceinline__ size_t packed_floats(int dim, int vp) {
    return (size_t)kChunkTokens * (3 * dim + vp);
}

struct RetChunk {
    int seq, begin, first, start, count;  // of the batch; first token among the step's of the sequence; its row; position; tokens
};
__device__ __forceinline__ RetChunk ret_chunk(const int* chunks, const int* seq_first_row, const int* seq_start,
                                              const int* seq_count, int c) {
    RetChunk m;
    m.seq = chunks[2 * c];
    m.begin = chunks[2 * c + 1];
    m.first = seq_first_row[m.seq] + m.begin;
    m.start = seq_start[m.seq] + m.begin;
    m.count = min(kChunkTokens, seq_count[m.seq] - m.begin);
    return m;
}

// g^0 .. g^64 as a chain of products; every thread of the block calls it
__device__ __forceinline__ void decay_powers(float g, float* pw) {
    if (threadIdx.x == 0) {
        float p = 1.f;
        for (int n = 0; n <= kChunkTokens; ++n) {
            pw[n] = p;
            p *= g;
        }
    }
    __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(256)
retention_pack_kernel(const T* __restrict__ qkvg, const float* __restrict__ freq, const float* __restrict__ decay,
                      const int* __restrict__ chunks, const int* __restrict__ seq_first_row,
                      const int* __restrict__ seq_start, const int* __restrict__ seq_count, float* __restrict__ packed,
                      int heads, int dim, int vdim, int vp, int rot_dims, int act, float k_scale) {
    constexpr int C = kChunkTokens;
    extern __shared__ float pack_smem[];
    __shared__ float pw[C + 1];
    pdl_wait();
    pdl_launch_dependents();
    const int ld = dim + 1, tid = threadIdx.x, h = blockIdx.y;
    float* qs = pack_smem;    // [64][dim + 1]
    float* ks = qs + C * ld;  // [64][dim + 1]
    const RetChunk ch = ret_chunk(chunks, seq_first_row, seq_start, seq_count, blockIdx.x);
    const size_t row_len = (size_t)2 * heads * (dim + vdim);
    const T* rows = qkvg + (size_t)ch.first * row_len + (size_t)h * dim;
    for (int it = tid; it < C * dim; it += 256) {
        const int t = it / dim, d = it - t * dim;
        const bool in = t < ch.count;
        qs[t * ld + d] = in ? pre(rows[(size_t)t * row_len + d], act) : 0.f;
        ks[t * ld + d] = in ? pre(rows[(size_t)t * row_len + (size_t)heads * dim + d], act) * k_scale : 0.f;
    }
    decay_powers(decay[h], pw);
    const int half = rot_dims >> 1;
    for (int it = tid; it < C * half; it += 256) {
        const int t = it & (C - 1), j = it >> 6;
        const float ang = (float)(ch.start + t) * freq[j];
        const float c = cosf(ang), sn = sinf(ang);
        float* q = qs + t * ld + j;
        float* k = ks + t * ld + j;
        const float q0 = q[0], q1 = q[half], k0 = k[0], k1 = k[half];
        q[0] = q0 * c - q1 * sn;
        q[half] = q1 * c + q0 * sn;
        k[0] = k0 * c - k1 * sn;
        k[half] = k1 * c + k0 * sn;
    }
    __syncthreads();
    float* to = packed + ((size_t)blockIdx.x * heads + h) * packed_floats(dim, vp);
    for (int it = tid; it < C * dim; it += 256) {
        const int t = it & (C - 1), d = it >> 6;
        to[it] = qs[t * ld + d];
        to[C * dim + it] = ks[t * ld + d];
    }
    to += (size_t)2 * C * dim;
    for (int it = tid; it < C * dim; it += 256) {
        const int t = it / dim, d = it - t * dim;
        to[it] = t < ch.count ? ks[t * ld + d] * pw[ch.count - 1 - t] : 0.f;
    }
    to += (size_t)C * dim;
    const T* v = qkvg + (size_t)ch.first * row_len + (size_t)2 * heads * dim + (size_t)h * vdim;
    for (int it = tid; it < C * vp; it += 256) {
        const int t = it / vp, j = it - t * vp;
        to[it] = t < ch.count && j < vdim ? pre(v[(size_t)t * row_len + j], act) : 0.f;
    }
}

template <int BV>
__global__ void __launch_bounds__(128)
retention_update_kernel(const float* __restrict__ packed, float* __restrict__ chunk_state, int heads, int dim, int vp) {
    extern __shared__ __align__(16) float update_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const int v_tiles = (vp + BV - 1) / BV;
    const size_t unit = (size_t)blockIdx.x * heads + blockIdx.y;
    const float* from = packed + unit * packed_floats(dim, vp) + (size_t)2 * kChunkTokens * dim;
    chunk_update_tile<BV>(from, from + (size_t)kChunkTokens * dim, chunk_state + unit * dim * vp, dim, vp,
                          (int)(blockIdx.z / v_tiles) * 64, (int)(blockIdx.z % v_tiles) * BV, update_smem);
}

// The chunk at which the scratch of a wave of pairs begins.
__device__ __forceinline__ int wave_chunk(const int* seq_first_chunk, int n_seqs, int pair0) {
    return pair0 ? find_chunk_pair(seq_first_chunk, n_seqs, pair0).chunk : 0;
}

// The state before every chunk in place of what the chunk adds, in order, a thread per four values of a row, eight
// chunks fetched ahead; the state after the last goes to the slot (whose rows have vdim values and no alignment).  The
// wave's chunks: `wave_n` from `wave0` on, the first of which chunk_state begins with; `by` = 2: pairs of chunks, each of which
// has added as one.
__global__ void __launch_bounds__(128)
retention_carry_kernel(float* chunk_state, float* state, const float* __restrict__ decay,
                       const int* __restrict__ seq_slots, const int* __restrict__ seq_start,
                       const int* __restrict__ seq_count, const int* __restrict__ seq_first_chunk, int wave0, int wave_n,
                       int heads, int dim, int vdim, int vp, int by) {
    constexpr int AHEAD = 8;
    pdl_wait();
    pdl_launch_dependents();
    const int seq = blockIdx.x, h = blockIdx.y, quads = vp >> 2;
    const int e = blockIdx.z * 128 + threadIdx.x;
    const int d = e / quads, j = (e - d * quads) * 4;
    const int begin = seq_first_chunk[seq], end = seq_first_chunk[seq + 1], count = seq_count[seq];
    int base = wave0, c0 = max(begin, wave0), c1 = min(end, wave0 + wave_n);
    if (by == 2) {
        const int pairs = chunk_pairs_before(seq_first_chunk, seq);
        base = wave_chunk(seq_first_chunk, gridDim.x, wave0);
        c0 = begin + 2 * max(wave0 - pairs, 0);
        c1 = min(end, begin + 2 * max(wave0 + wave_n - pairs, 0));
    }
    if (c1 <= c0 || e >= dim * quads) return;
    const float g = decay[h];
    float g_chunk = 1.f, g_last = 1.f;  // as decay_powers makes them
    const int last = count - (end - begin - 1) * kChunkTokens;
    for (int n = 0; n < kChunkTokens; ++n) {
        g_chunk *= g;
        if (n < last) g_last *= g;
    }
    float* own = chunk_state + ((size_t)(c0 - base) * heads + h) * dim * vp + (size_t)d * vp + j;
    const size_t step = (size_t)heads * dim * vp;
    float* slot = state + ((size_t)seq_slots[seq] * heads + h) * dim * vdim + (size_t)d * vdim + j;
    float run[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) run[v] = j + v < vdim ? slot[v] : 0.f;
    for (int c = c0; c < c1; c += AHEAD * by) {
        float4 add[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (c + k * by < c1) add[k] = load4(own + (size_t)(c - c0 + k * by) * step);
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int at = c + k * by, past = min(at + by, c1);
            if (at >= c1) break;
            store4(own + (size_t)(at - c0) * step, make_float4(run[0], run[1], run[2], run[3]));
            const float f = (past == end ? g_last : g_chunk) * (past - at == 2 ? g_chunk : 1.f);
            run[0] = fmaf(f, run[0], add[k].x);
            run[1] = fmaf(f, run[1], add[k].y);
            run[2] = fmaf(f, run[2], add[k].z);
            run[3] = fmaf(f, run[3], add[k].w);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
        if (j + v < vdim) slot[v] = run[v];
}

template <int BV>
__global__ void __launch_bounds__(128, 3)
retention_read_kernel(const float* __restrict__ packed, const float* __restrict__ chunk_state,
                      const float* __restrict__ decay, const int* __restrict__ chunks,
                      const int* __restrict__ seq_first_row, const int* __restrict__ seq_start,
                      const int* __restrict__ seq_count, float* __restrict__ o_raw, int heads, int dim, int vdim, int vp) {
    extern __shared__ __align__(16) float read_smem[];
    __shared__ float pw[kChunkTokens + 1];
    pdl_wait();
    pdl_launch_dependents();
    const int h = blockIdx.y, v0 = blockIdx.z * BV;
    const RetChunk ch = ret_chunk(chunks, seq_first_row, seq_start, seq_count, blockIdx.x);
    decay_powers(decay[h], pw);
    const size_t unit = (size_t)blockIdx.x * heads + h;
    const float* q = packed + unit * packed_floats(dim, vp);
    unsigned long long acc[8][BV / 32];
    chunk_read_tile<BV>(q, q + (size_t)kChunkTokens * dim, ch.start > 0 ? chunk_state + unit * dim * vp : nullptr,
                        q + (size_t)3 * kChunkTokens * dim, dim, vp, v0, ch.count, read_smem, acc,
                        [&](int i, int j, float x) { return j <= i ? x * pw[i - j] : 0.f; },
                        [&](int i) { return pw[i + 1]; });
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const bool whole = (vdim & 3) == 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int t = ty * 8 + r;
        if (t >= ch.count) continue;
        float* row = o_raw + ((size_t)(ch.first + t) * heads + h) * vdim;
#pragma unroll
        for (int c = 0; c < BV / 64; ++c) {
            const int j = v0 + c * 64 + tx * 4;
            const float2 a = halves(acc[r][2 * c]), b = halves(acc[r][2 * c + 1]);
            if (whole) {
                if (j < vdim) store4(row + j, make_float4(a.x, a.y, b.x, b.y));
            } else {
                const float x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j + e < vdim) row[j + e] = x[e];
            }
        }
    }
}

// Keys of 64 and 128, values in whole groups of eight: `update` and `read` by pairs of chunks on the tensor cores, where
// retention_by_pairs says so.  A wave holds whole pairs, so that results have the same
// bits however many fit it; its first chunk is the one at which the scratch begins.  A packed
// (chunk, head) is then queries [64][dim], keys [64][dim] and values [64][vdim], rows of tokens that are not there left alone;
// four CTAs a (chunk, head), 16 tokens each: 2,048 tokens, eight heads of 128 x 256, 37 -> 16 us (three layouts and powers of the
// decay made by one thread before).
template <typename T>
__global__ void __launch_bounds__(256)
retention_pack_rows_kernel(const T* __restrict__ qkvg, const float* __restrict__ freq, const int* __restrict__ chunks,
                           const int* __restrict__ seq_first_row, const int* __restrict__ seq_start,
                           const int* __restrict__ seq_count, float* __restrict__ packed, int heads, int dim, int vdim,
                           int rot_dims, int act, float k_scale, const int* __restrict__ seq_first_chunk, int n_seqs,
                           int pair0) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int TOKENS = kChunkTokens / 4;
    const int h = blockIdx.y, t0 = blockIdx.z * TOKENS, tid = threadIdx.x;
    const ChunkPair pair = find_chunk_pair(seq_first_chunk, n_seqs, pair0 + (int)blockIdx.x / 2);
    const int c = pair.chunk + (int)(blockIdx.x & 1);
    if (pair.seq < 0 || c >= seq_first_chunk[pair.seq + 1]) return;
    const size_t unit = (size_t)(c - wave_chunk(seq_first_chunk, n_seqs, pair0)) * heads + h;
    const RetChunk ch = ret_chunk(chunks, seq_first_row, seq_start, seq_count, c);
    const int there = min(TOKENS, ch.count - t0);
    if (there <= 0) return;
    const size_t row_len = (size_t)2 * heads * (dim + vdim);
    const T* q = qkvg + (size_t)(ch.first + t0) * row_len + (size_t)h * dim;
    const T* k = q + (size_t)heads * dim;
    const T* v = qkvg + (size_t)(ch.first + t0) * row_len + (size_t)2 * heads * dim + (size_t)h * vdim;
    float* qt = packed + unit * packed_floats(dim, vdim) + (size_t)t0 * dim;
    float* kt = qt + (size_t)kChunkTokens * dim;
    float* vt = qt + (size_t)2 * kChunkTokens * dim - (size_t)t0 * dim + (size_t)t0 * vdim;
    const int half = rot_dims >> 1, rest = dim - rot_dims;
    for (int it = tid; it < there * half; it += 256) {
        const int t = it / half, j = it - t * half;
        const T *qr = q + t * row_len + j, *kr = k + t * row_len + j;
        const float q0 = pre(qr[0], act), q1 = pre(qr[half], act);
        const float k0 = pre(kr[0], act) * k_scale, k1 = pre(kr[half], act) * k_scale;
        const float ang = (float)(ch.start + t0 + t) * freq[j];
        const float c = cosf(ang), sn = sinf(ang);
        qt[t * dim + j] = q0 * c - q1 * sn;
        qt[t * dim + j + half] = q1 * c + q0 * sn;
        kt[t * dim + j] = k0 * c - k1 * sn;
        kt[t * dim + j + half] = k1 * c + k0 * sn;
    }
    for (int it = tid; it < there * rest; it += 256) {
        const int t = it / rest, j = rot_dims + it - t * rest;
        qt[t * dim + j] = pre(q[t * row_len + j], act);
        kt[t * dim + j] = pre(k[t * row_len + j], act) * k_scale;
    }
    const int quads = vdim >> 2;
    for (int it = tid; it < there * quads; it += 256) {
        const int t = it / quads, j = (it - t * quads) * 4;
        float4 x = load4(v + t * row_len + j);
        if (act) x = make_float4(pre(x.x, 1), pre(x.y, 1), pre(x.z, 1), pre(x.w, 1));
        store4(vt + (size_t)t * vdim + j, x);
    }
}

struct RetPair {
    int seq, first, start, count;  // of the first chunk: row, position; tokens of both
    ChunkReadRows rows;
};
__device__ __forceinline__ RetPair ret_pair(const float* packed, const int* seq_first_chunk, int n_seqs, int pair0, const int* seq_first_row,
                                            const int* seq_start, const int* seq_count, int heads,
                                            int dim, int vdim, int cols, size_t& unit) {
    const ChunkPair at = find_chunk_pair(seq_first_chunk, n_seqs, pair0 + (int)blockIdx.x);
    RetPair p;
    p.seq = at.seq;
    if (at.seq < 0) return p;
    const int begin = (at.chunk - seq_first_chunk[at.seq]) * kChunkTokens, v0 = blockIdx.z * cols;
    p.first = seq_first_row[at.seq] + begin;
    p.start = seq_start[at.seq] + begin;
    p.count = min(2 * kChunkTokens, seq_count[at.seq] - begin);
    unit = (size_t)(at.chunk - wave_chunk(seq_first_chunk, n_seqs, pair0)) * heads + blockIdx.y;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        p.rows.q[i] = packed + (unit + (size_t)i * heads) * packed_floats(dim, vdim);
        p.rows.k[i] = p.rows.q[i] + (size_t)kChunkTokens * dim;
        p.rows.v[i] = p.rows.k[i] + (size_t)kChunkTokens * dim + v0;
    }
    p.rows.q_stride = p.rows.k_stride = dim;
    p.rows.v_stride = p.rows.state_stride = vdim;
    p.rows.state = nullptr;
    p.rows.count = p.count;
    p.rows.dim = dim;
    p.rows.cols = min(cols, vdim - v0);
    p.rows.q_scale = 1.f;
    return p;
}
// g^0 .. g^128: the second chunk's as what a state that passes the first one's end is multiplied by
__device__ __forceinline__ void decay_powers_of_pairs(float g, float* pw) {
    decay_powers(g, pw);
    if (threadIdx.x > 0 && threadIdx.x <= kChunkTokens) pw[kChunkTokens + threadIdx.x] = pw[kChunkTokens] * pw[threadIdx.x];
    __syncthreads();
}

// 2,048 tokens, eight heads of 128 x 256: 25 -> 16 us, and retention_carry, with half the sums to walk, 12 -> 8 us.
__global__ void __launch_bounds__(kCrThreads, 1)
retention_update_split_kernel(const float* __restrict__ packed, float* __restrict__ chunk_state,
                              const float* __restrict__ decay, const int* __restrict__ seq_first_chunk, int n_seqs,
                              int pair0, const int* __restrict__ seq_first_row,
                              const int* __restrict__ seq_start, const int* __restrict__ seq_count, int heads, int dim,
                              int vdim, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char sum_smem[];
    __shared__ ChunkReadShared sh;
    __shared__ float pw[2 * kChunkTokens + 1];
    pdl_wait();
    pdl_launch_dependents();
    constexpr int COLS = kCrTiles * kCrCols;
    size_t unit = 0;
    const RetPair p = ret_pair(packed, seq_first_chunk, n_seqs, pair0, seq_first_row, seq_start, seq_count, heads, dim, vdim,
                               COLS, unit);
    if (p.seq < 0) return;
    float* to = chunk_state + unit * dim * vdim + blockIdx.z * COLS;
    chunk_sum_split(
        p.rows, nullptr, sh, sum_smem, status, [&] { decay_powers_of_pairs(decay[blockIdx.y], pw); },
        [&](int t) { return t < p.count ? pw[p.count - 1 - t] : 0.f; },
        [&](int d, int c, const float* x) { store8(to + (size_t)d * vdim + c, x); });
}

// 2,048 tokens, eight heads of 128 x 256: 66 -> 30 us.
__global__ void __launch_bounds__(kCrThreads, 1)
retention_read_split_kernel(const float* __restrict__ packed, const float* __restrict__ chunk_state,
                            const float* __restrict__ decay, const int* __restrict__ seq_first_chunk, int n_seqs, int pair0,
                            const int* __restrict__ seq_first_row, const int* __restrict__ seq_start,
                            const int* __restrict__ seq_count, float* __restrict__ o_raw, int heads, int dim, int vdim,
                            int cols, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char read_smem_split[];
    __shared__ ChunkReadShared sh;
    __shared__ float pw[2 * kChunkTokens + 1];
    pdl_wait();
    pdl_launch_dependents();
    size_t unit = 0;
    RetPair p = ret_pair(packed, seq_first_chunk, n_seqs, pair0, seq_first_row, seq_start, seq_count, heads, dim, vdim, cols,
                         unit);
    if (p.seq < 0) return;
    const int h = blockIdx.y, v0 = blockIdx.z * cols;
    if (p.start > 0) p.rows.state = chunk_state + unit * dim * vdim + v0;
    chunk_read_split(
        p.rows, nullptr, sh, read_smem_split, status, [&] { decay_powers_of_pairs(decay[h], pw); },
        [&](int i, int j, float x) { return x * pw[i - j]; }, [&](int i) { return pw[i + 1]; },
        [&](int i, int c, const float* x, float, float) {
            store8(o_raw + ((size_t)(p.first + i) * heads + h) * vdim + v0 + c, x);
        });
}

// Whether chunks go by pairs: not for heads of 64 x 64 and smaller unless there is a CTA for two SMs of three and
// sequences are long, as most of a tile of 128 columns is padding (8 heads of 64 x 64, us by pairs and by single chunks:
// 512 tokens 37, 35, 16 x 130 66, 58, 40 x 70 95, 81; 1,000 40, 50, 4 x 400 43, 53, 4,000 79, 86; of 64 x 32 512 36, 34,
// 1,000 39, 49).  With 128 keys they win with few values too (8 heads of 128 x 8: 512 tokens 42, 54, 16 x 130 71, 79,
// 4,000 89, 124).
static bool retention_by_pairs(long long n_chunks, long long n_seqs, int heads, int dim, int vdim, int wave) {
    if (vdim % 8 || (wave < 2 && n_chunks > 1)) return false;
    return dim == 128 || (dim == 64 && (vdim > 64 || (n_chunks * heads >= 100 && n_chunks >= 4 * n_seqs)));
}
// Pairs: at most as many, and as many as the scratch holds at a time.
static int retention_pairs(int n_chunks, int n_seqs) { return (n_chunks + n_seqs) / 2; }
static int retention_pairs_held(int n_chunks, int n_seqs, int wave) {
    return n_chunks <= wave ? retention_pairs(n_chunks, n_seqs) : wave / 2;
}

template <typename T>
static int launch_chunks(const T* qkvg, const float* freq, const float* decay, float* state, const int* seq_slots,
                         const int* seq_first_row, const int* seq_start, const int* seq_count, const int* chunks,
                         int n_chunks, const int* seq_first_chunk, int wave, float* packed, float* chunk_state, float* o_raw,
                         int n_seqs, int heads, int dim, int vdim, int rot_dims, int act, float k_scale, int sms, int* status,
                         cudaStream_t stream) {
    // (rows of q, k and v in whole groups of eight on 16-byte borders, float32 rows on 32-byte borders)
    if (retention_by_pairs(n_chunks, n_seqs, heads, dim, vdim, wave) && (uintptr_t)qkvg % 16 == 0 &&
        ((uintptr_t)packed | (uintptr_t)chunk_state | (uintptr_t)o_raw) % 32 == 0) {
        cudaError_t e = cudaFuncSetAttribute(retention_update_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCrSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(retention_read_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCrSmem);
        const int all = retention_pairs(n_chunks, n_seqs), most = kCrTiles * kCrCols;
        const int held = retention_pairs_held(n_chunks, n_seqs, wave);
        for (int p0 = 0; p0 < all && e == cudaSuccess; p0 += held) {
            const int n = all - p0 < held ? all - p0 : held, cols = chunk_read_cols((long long)n * heads, vdim, sms);
            e = launch_dependent(retention_pack_rows_kernel<T>, dim3(2 * n, heads, 4), 256, 0, stream, qkvg, freq, chunks,
                                 seq_first_row, seq_start, seq_count, packed, heads, dim, vdim, rot_dims, act, k_scale,
                                 seq_first_chunk, n_seqs, p0);
            if (e == cudaSuccess)
                e = launch_dependent(retention_update_split_kernel, dim3(n, heads, (vdim + most - 1) / most), kCrThreads,
                                     kCrSmem, stream, (const float*)packed, chunk_state, decay, seq_first_chunk, n_seqs, p0,
                                     seq_first_row, seq_start, seq_count, heads, dim, vdim, status);
            if (e == cudaSuccess)
                e = launch_dependent(retention_carry_kernel, dim3(n_seqs, heads, (dim * (vdim / 4) + 127) / 128), 128, 0,
                                     stream, chunk_state, state, decay, seq_slots, seq_start, seq_count, seq_first_chunk, p0,
                                     n, heads, dim, vdim, vdim, 2);
            if (e == cudaSuccess)
                e = launch_dependent(retention_read_split_kernel, dim3(n, heads, (vdim + cols - 1) / cols), kCrThreads,
                                     kCrSmem, stream, (const float*)packed, (const float*)chunk_state, decay, seq_first_chunk,
                                     n_seqs, p0, seq_first_row, seq_start, seq_count, o_raw, heads, dim, vdim, cols, status);
        }
        return e == cudaSuccess ? NNIS_OK : (int)e;
    }
    const int vp = (vdim + 3) & ~3, bv = vp > 64 ? 128 : 64;
    const int pack_smem = 2 * kChunkTokens * (dim + 1) * 4, update_smem = kChunkTokens * (64 + bv) * 4;
    const int read_smem = (bv == 128 ? chunk_read_floats<128>() : chunk_read_floats<64>()) * 4;
    auto update = bv == 128 ? retention_update_kernel<128> : retention_update_kernel<64>;
    auto read = bv == 128 ? retention_read_kernel<128> : retention_read_kernel<64>;
    cudaError_t e = cudaFuncSetAttribute(retention_pack_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, pack_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(update, cudaFuncAttributeMaxDynamicSharedMemorySize, update_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(read, cudaFuncAttributeMaxDynamicSharedMemorySize, read_smem);
    const int v_tiles = (vp + bv - 1) / bv;
    for (int c0 = 0; c0 < n_chunks && e == cudaSuccess; c0 += wave) {
        const int n = n_chunks - c0 < wave ? n_chunks - c0 : wave;
        const int* own = chunks + 2 * c0;
        e = launch_dependent(retention_pack_kernel<T>, dim3(n, heads), 256, pack_smem, stream, qkvg, freq, decay, own,
                             seq_first_row, seq_start, seq_count, packed, heads, dim, vdim, vp, rot_dims, act, k_scale);
        if (e == cudaSuccess)
            e = launch_dependent(update, dim3(n, heads, (dim + 63) / 64 * v_tiles), 128, update_smem, stream,
                                 (const float*)packed, chunk_state, heads, dim, vp);
        if (e == cudaSuccess)
            e = launch_dependent(retention_carry_kernel, dim3(n_seqs, heads, (dim * (vp / 4) + 127) / 128), 128, 0, stream,
                                 chunk_state, state, decay, seq_slots, seq_start, seq_count, seq_first_chunk, c0, n, heads,
                                 dim, vdim, vp, 1);
        if (e == cudaSuccess)
            e = launch_dependent(read, dim3(n, heads, v_tiles), 128, read_smem, stream, (const float*)packed,
                                 (const float*)chunk_state, decay, own, seq_first_row, seq_start, seq_count, o_raw, heads,
                                 dim, vdim, vp);
    }
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

// out[n, h, :] = o[n, h, :] / sqrt(mean(o[n, h, :]^2) + eps) * silu(g[n, h, :]); a warp
// per (token, head); a row at position -1 is left alone
template <typename T>
__global__ void __launch_bounds__(256)
retention_gate_kernel(const float* __restrict__ o_raw, const T* __restrict__ qkvg,
                      const int* __restrict__ token_pos, T* __restrict__ out, long long n_units,
                      int heads, int dim, int vdim, float eps, int gate_kind) {
    pdl_wait();
    pdl_launch_dependents();
    long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= n_units) return;
    int lane = threadIdx.x & 31;
    long long n = unit / heads;
    int h = (int)(unit - n * heads);
    T* dst = out + (size_t)unit * vdim;
    if (token_pos[n] < 0) {
        for (int i = lane; i < vdim; i += 32) dst[i] = from_float<T>(0.f);
        return;
    }
    const float* o = o_raw + (size_t)unit * vdim;
    const T* gate = qkvg + (size_t)n * ((size_t)2 * heads * dim + (size_t)2 * heads * vdim) +
                    (size_t)2 * heads * dim + (size_t)heads * vdim + (size_t)h * vdim;
    float ss = 0.f;
    for (int i = lane; i < vdim; i += 32) ss = fmaf(o[i], o[i], ss);
    ss = warp_sum(ss);
    float s = 1.0f / sqrtf(ss / (float)vdim + eps);
    for (int i = lane; i < vdim; i += 32) {
        float z = to_float(gate[i]);
        float sg = 1.0f / (1.0f + expf(-z));
        dst[i] = from_float<T>((o[i] * s) * (gate_kind ? sg : z * sg));
    }
}

// The same for heads of a multiple of four values, at most 128 Q, with rows on 16-byte borders.
template <typename T, int Q>
__global__ void __launch_bounds__(256)
retention_gate_quads_kernel(const float* __restrict__ o_raw, const T* __restrict__ qkvg,
                            const int* __restrict__ token_pos, T* __restrict__ out, long long n_units,
                            int heads, int dim, int vdim, float eps, int gate_kind) {
    pdl_wait();
    pdl_launch_dependents();
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= n_units) return;
    const int lane = threadIdx.x & 31, n4 = vdim >> 2;
    const long long n = unit / heads;
    T* dst = out + (size_t)unit * vdim;
    if (token_pos[n] < 0) {
        for (int i = lane; i < n4; i += 32) store4(dst + 4 * i, make_float4(0.f, 0.f, 0.f, 0.f));
        return;
    }
    const T* gate = qkvg + (size_t)n * ((size_t)2 * heads * (dim + vdim)) + (size_t)2 * heads * dim +
                    (size_t)heads * vdim + (size_t)(unit - n * heads) * vdim;
    finish_head<T, Q>(o_raw + (size_t)unit * vdim, dst, n4, eps, lane, [&](int i) {
        const float4 z = load4(gate + 4 * i);
        const float4 s = make_float4(1.0f / (1.0f + expf(-z.x)), 1.0f / (1.0f + expf(-z.y)), 1.0f / (1.0f + expf(-z.z)),
                                     1.0f / (1.0f + expf(-z.w)));
        return gate_kind ? s : make_float4(z.x * s.x, z.y * s.y, z.z * s.z, z.w * s.w);
    });
}

template <typename T>
static auto retention_gate_of(const float* o_raw, const T* qkvg, const T* out, int heads, int dim, int vdim) {
    const bool quads = vdim % 4 == 0 && vdim <= 512 && (2 * heads * dim) % 4 == 0 &&
                       ((uintptr_t)o_raw | (uintptr_t)qkvg | (uintptr_t)out) % 16 == 0;
    return !quads ? retention_gate_kernel<T> : vdim <= 128 ? retention_gate_quads_kernel<T, 1>
           : vdim <= 256 ? retention_gate_quads_kernel<T, 2> : retention_gate_quads_kernel<T, 4>;
}

// The same with ONE norm over the joined heads of a token and a weight per value:
// out[n, :] = o[n, :] / sqrt(mean(o[n, :]^2) + eps) * w * gate(g[n, :]); a CTA per token
template <typename T>
__global__ void __launch_bounds__(256)
retention_gate_joined_kernel(const float* __restrict__ o_raw, const T* __restrict__ qkvg,
                             const float* __restrict__ w, const int* __restrict__ token_pos, T* __restrict__ out,
                             int heads, int dim, int vdim, float eps, int gate_kind) {
    __shared__ float red[8];
    pdl_wait();
    pdl_launch_dependents();
    const size_t n = blockIdx.x;
    const int cols = heads * vdim;
    T* dst = out + n * cols;
    if (token_pos[n] < 0) {
        for (int i = threadIdx.x; i < cols; i += 256) dst[i] = from_float<T>(0.f);
        return;
    }
    const float* o = o_raw + n * cols;
    const T* gate = qkvg + n * ((size_t)2 * heads * dim + (size_t)2 * cols) + (size_t)2 * heads * dim + cols;
    float ss = 0.f;
    for (int i = threadIdx.x; i < cols; i += 256) ss = fmaf(o[i], o[i], ss);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) total += red[k];
    const float s = 1.0f / sqrtf(total / (float)cols + eps);
    for (int i = threadIdx.x; i < cols; i += 256) {
        float z = to_float(gate[i]);
        float sg = 1.0f / (1.0f + expf(-z));
        dst[i] = from_float<T>((o[i] * s) * w[i] * (gate_kind ? sg : z * sg));
    }
}

template <typename T>
static int launch_retention(const void* qkvg, const float* freq, const float* decay, float* state,
                            const int* token_pos, const int* token_seq, const int* seq_slots,
                            const int* seq_first_row, const int* seq_start, const int* seq_count,
                            const int* chunks, int n_chunks, const int* seq_first_chunk, int wave, float* packed,
                            float* chunk_state, float* o_raw, void* out, int n_tokens, int n_units, int heads, int dim,
                            int vdim, int rot_dims, float eps, int act, float k_scale, const float* norm_w,
                            int gate_kind, int sms, int* status, cudaStream_t stream) {
    dim3 grid(n_units, heads, (vdim + 31) / 32);
    cudaError_t le = cudaSuccess;
    if (chunks) {  // a prompt step, chunks of tokens side by side
        int rc = launch_chunks<T>((const T*)qkvg, freq, decay, state, seq_slots, seq_first_row, seq_start, seq_count,
                                  chunks, n_chunks, seq_first_chunk, wave, packed, chunk_state, o_raw, n_units, heads, dim,
                                  vdim, rot_dims, act, k_scale, sms, status, stream);
        if (rc != NNIS_OK) return rc;
    } else if (seq_first_row && (dim == 32 || dim == 64 || dim == 128 || dim == 256)) {
        constexpr int C = kRetChunk;
        const size_t smem = (2 * (size_t)C * (dim + 4) + (size_t)dim * 32 + C * (C + 1) + C * 32 + C + 1) * sizeof(float);
        auto kernel = dim == 32 ? retention_in_order_kernel<T, 1> : dim == 64 ? retention_in_order_kernel<T, 2>
                      : dim == 128 ? retention_in_order_kernel<T, 4> : retention_in_order_kernel<T, 8>;
        le = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (le != cudaSuccess) return (int)le;
        kernel<<<grid, 256, smem, stream>>>((const T*)qkvg, freq, decay, state, seq_slots, seq_first_row, seq_start,
                                            seq_count, o_raw, heads, vdim, rot_dims, act, k_scale);
        le = cudaGetLastError();
        if (le != cudaSuccess) return (int)le;
    } else {
        size_t smem = (2 * (size_t)dim + 256) * sizeof(float);
#define NNIS_RET_CASE(R) \
        le = launch_dependent(retention_scan_kernel<T, R>, grid, 256, smem, stream, (const T*)qkvg, freq, decay, state, \
                              token_pos, token_seq, seq_slots, seq_first_row, seq_start, seq_count, o_raw, heads, dim, \
                              vdim, rot_dims, act, k_scale)
        if (dim <= 32) NNIS_RET_CASE(4);
        else if (dim <= 64) NNIS_RET_CASE(8);
        else if (dim <= 128) NNIS_RET_CASE(16);
        else NNIS_RET_CASE(32);
#undef NNIS_RET_CASE
        if (le != cudaSuccess) return (int)le;
    }
    if (norm_w) {
        le = launch_dependent(retention_gate_joined_kernel<T>, (unsigned)n_tokens, 256, 0, stream,
                              (const float*)o_raw, (const T*)qkvg, norm_w, token_pos, (T*)out, heads, dim, vdim, eps,
                              gate_kind);
        return le == cudaSuccess ? NNIS_OK : (int)le;
    }
    long long units = (long long)n_tokens * heads;
    le = launch_dependent(retention_gate_of<T>(o_raw, (const T*)qkvg, (const T*)out, heads, dim, vdim), (unsigned)((units + 7) / 8), 256, 0, stream,
                          (const float*)o_raw, (const T*)qkvg, token_pos, (T*)out, units, heads, dim, vdim, eps,
                          gate_kind);
    return le == cudaSuccess ? NNIS_OK : (int)le;
}

}  // namespace nnis

using namespace nnis;

// Kernels that a prompt step of these sizes launches, chunks side by side (qkvg on 16-byte, the scratch and o_raw on 32-byte
// boundaries).
NNIS_API int nnis_retention_launches(int n_chunks, int n_seqs, int heads, int dim, int vdim, int wave) {
    if (!retention_by_pairs(n_chunks, n_seqs, heads, dim, vdim, wave)) return 4 * ((n_chunks + wave - 1) / wave) + 1;
    const int all = retention_pairs(n_chunks, n_seqs), held = retention_pairs_held(n_chunks, n_seqs, wave);
    return 4 * ((all + held - 1) / held) + 1;
}

// `seq_first_row` null: every row is a sequence of its own bringing one token
// (`n_units` = n_tokens); else `n_units` sequences with their first row, first
// position and token count.  `o_raw`: float32 scratch [n_tokens, heads * vdim].
// `chunks` (prompt steps, key sizes 32, 64, 128 and 256; without it the tokens are worked in order): int32
// [n_chunks, 2] = (sequence, first token of the chunk among the sequence's tokens of this step), 64 tokens each in the
// order of the sequences, with `seq_first_chunk` [n_units + 1] and, vp = vdim rounded up to a multiple of four, float32
// scratch `packed` [wave, heads, 64 (3 dim + vp)] and `chunk_state` [wave, heads, dim, vp] (of n_chunks, if these are
// fewer): `wave` chunks are worked at a time.
// `act` 1: q, k, v through silu; `k_scale`: the keys' multiplier; `norm_w` (float32 [heads * vdim]): one
// norm over the joined heads with this weight instead of a norm per head; `gate_kind` 0 silu, 1 sigmoid.
NNIS_API int nnis_retention(const void* qkvg, const float* freq, const float* decay, float* state,
                            const int* token_pos, const int* token_seq, const int* seq_slots,
                            const int* seq_first_row, const int* seq_start, const int* seq_count,
                            const int* chunks, int n_chunks, const int* seq_first_chunk, int wave, float* packed,
                            float* chunk_state, float* o_raw, void* out, int n_tokens, int n_units, int heads, int dim,
                            int vdim, int rot_dims, float eps, int act, float k_scale, const float* norm_w,
                            int gate_kind, int dtype, int sms, int* status, cudaStream_t stream) {
    if (n_tokens <= 0 || sms <= 0 || n_units <= 0 || heads <= 0 || dim <= 0 || vdim <= 0 || rot_dims < 0 ||
        (rot_dims & 1) || rot_dims > dim || !(eps > 0.f) || !qkvg || !freq || !decay || !state ||
        !token_pos || !token_seq || !seq_slots || !o_raw || !out)
        return NNIS_ERR_ARGUMENT;
    if (seq_first_row && (!seq_start || !seq_count)) return NNIS_ERR_ARGUMENT;
    if (chunks && (!seq_first_row || n_chunks <= 0 || wave <= 0 || !seq_first_chunk || !packed || !chunk_state ||
                   !(dim == 32 || dim == 64 || dim == 128 || dim == 256)))
        return NNIS_ERR_ARGUMENT;
    if (chunks && ((uintptr_t)packed | (uintptr_t)chunk_state | (uintptr_t)o_raw) % 16) return NNIS_ERR_ALIGNMENT;
    if (dim > 256 || heads > 65535 || (vdim + 31) / 32 > 65535) return NNIS_ERR_UNSUPPORTED;
    if (dtype == NNIS_DTYPE_F32)
        return launch_retention<float>(qkvg, freq, decay, state, token_pos, token_seq, seq_slots,
                                       seq_first_row, seq_start, seq_count, chunks, n_chunks,
                                       seq_first_chunk, wave, packed, chunk_state, o_raw, out, n_tokens, n_units, heads, dim, vdim, rot_dims, eps, act, k_scale, norm_w, gate_kind, sms, status, stream);
    if (dtype == NNIS_DTYPE_BF16)
        return launch_retention<bf16>(qkvg, freq, decay, state, token_pos, token_seq, seq_slots,
                                      seq_first_row, seq_start, seq_count, chunks, n_chunks,
                                      seq_first_chunk, wave, packed, chunk_state, o_raw, out, n_tokens, n_units, heads, dim, vdim, rot_dims, eps, act, k_scale, norm_w, gate_kind, sms, status, stream);
    return NNIS_ERR_UNSUPPORTED;
}
