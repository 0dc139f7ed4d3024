// The gated delta rule (delta_rule.cu) over a prompt, 64 tokens at a time.  With c_i the sum of the log decays of a
// chunk up to token i, S_0 the state before the chunk and u_i what token i writes,
//     S_i = e^(c_i) S_0 + sum_(j<=i) e^(c_i - c_j) k_j u_j^T
//     u_i + sum_(j<i) beta_i e^(c_i - c_j) (k_i . k_j) u_j = beta_i (v_i - e^(c_i) S_0^T k_i)
//     o_i = e^(c_i) S_0^T q_i + sum_(j<=i) e^(c_i - c_j) (q_i . k_j) u_j
// so a chunk is a unit lower triangular system with two right sides, U = U0 - W S_0, and products:
//   delta_pack    convolution, silu, unit vectors, beta and c of every chunk, in the layouts that the products read;
//   delta_solve   a CTA per (chunk, head), all side by side: k_i . k_j, then W and U0 by forward substitution, two
//                 columns a thread in registers;
//   delta_chain   a CTA per (sequence, head, 32 columns) walks the chunks: U = U0 - W S, S <- e^c S + K^T (e^(c - c_j) U);
//                 it leaves U and the state before every chunk;
//   delta_read    a CTA per (chunk, head, columns), all side by side: the outputs (linear_chunks.cuh).
// More chunks than the scratch holds go through the four kernels in waves, the slot's state from one to the next (the same
// bits: the state is float32 there too).
// Everything is float32 with fmaf on the CUDA cores; c is double (differences of sums of up to 64 logs keep float32's
// digits), a decay of zero counts as e^-200, which is zero in float32 and leaves the tokens after it exact.
//
// Against the walk in runs with a transition matrix per run (delta_rule.cu, which other key sizes and short prompts
// keep): a token costs 2.2 dim vdim + 64 (dim + vdim) multiply-adds or so instead of 2.3 times three dim vdim, all but the chain side
// by side, and a thread's 8 x 8 outputs share what is read.
// Two prompts of 2,048 and 555 tokens, 32 heads over 16 key heads of 128 x 128, on a B200: prep 201, walk 707, prefix 270
// and apply 235 us before; now pack 60, solve 147, chain 255 and read 133.
#include "async_copy.cuh"
#include "common.cuh"
#include "linear_chunks.cuh"

namespace nnis {

constexpr int kDC = kChunkTokens;
constexpr double kDeltaLeastLog = -200.0;

struct DeltaChunk {
    int seq, first, start, count;  // of the batch; the chunk's first row; tokens of the step before it; tokens
};
__device__ __forceinline__ DeltaChunk delta_chunk(const int* chunks, const int* seq_first_row, const int* seq_count, int c) {
    DeltaChunk m;
    m.seq = chunks[2 * c];
    m.start = chunks[2 * c + 1];
    m.first = seq_first_row[m.seq] + m.start;
    m.count = min(kDC, seq_count[m.seq] - m.start);
    return m;
}

// A packed (chunk, key head): queries [dim][64], keys [dim][64], keys [64][dim]; and (chunk, head): values [64][vp].
__host__ __device__ __forceinline__ size_t delta_qk_floats(int dim) { return (size_t)3 * kDC * dim; }

// A CTA per (chunk, piece): q heads, k heads, value heads, and last the gates of all heads.  A thread walks 16 tokens of
// a channel; with TAPS (the taps when there are 4, else 0) the inputs before a token stay in registers.  Instructions bound it
// (104 a value with a division for each place and a test for each input, 79 us on the prompts above; 60 us now).
template <int TAPS>
__global__ void __launch_bounds__(256)
delta_pack_kernel(const float* __restrict__ a, const float* __restrict__ conv_w, const float* __restrict__ tail,
                  const float* __restrict__ a_log, const float* __restrict__ dt_bias, const int* __restrict__ chunks,
                  const int* __restrict__ seq_slots, const int* __restrict__ seq_first_row,
                  const int* __restrict__ seq_count, float* __restrict__ qk, float* __restrict__ values,
                  float* __restrict__ beta, double* __restrict__ logs, int H, int G, int dim, int vdim, int vp,
                  int taps, float unit_eps, float q_scale) {
    extern __shared__ float pack_y[];  // [64][width + 1]
    __shared__ float scale[kDC];
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, piece = blockIdx.y;
    const DeltaChunk ch = delta_chunk(chunks, seq_first_row, seq_count, blockIdx.x);
    const int nqk = 2 * G * dim, conv_cols = nqk + H * vdim;
    const size_t row_len = (size_t)conv_cols + (size_t)H * vdim + 2 * H;
    if (piece == 2 * G + H) {
        for (int h = warp; h < H; h += 8) {
            double lg[2];
            float bt[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 2 * lane + e;
                lg[e] = 0.0;
                bt[e] = 0.f;
                if (t < ch.count) {
                    const float* g = a + (size_t)(ch.first + t) * row_len + conv_cols + (size_t)H * vdim;
                    bt[e] = 1.0f / (1.0f + expf(-g[h]));
                    const float x = g[H + h] + dt_bias[h];
                    const float decay = expf(-expf(a_log[h]) * (x > 20.f ? x : log1pf(expf(x))));
                    const double l = log((double)decay);
                    lg[e] = l < kDeltaLeastLog ? kDeltaLeastLog : l;  // (a decay that is no number stays one)
                }
            }
            double sum = lg[0] + lg[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double x = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += x;
            }
            double before = __shfl_up_sync(0xffffffffu, sum, 1);
            if (lane == 0) before = 0.0;
            const size_t at = ((size_t)blockIdx.x * H + h) * kDC + 2 * lane;
            beta[at] = bt[0];
            beta[at + 1] = bt[1];
            logs[at] = before + lg[0];
            logs[at + 1] = sum;
        }
        return;
    }
    const bool head = piece < 2 * G;
    const int width = head ? dim : vdim, c0 = head ? piece * dim : nqk + (piece - 2 * G) * vdim, ld = width + 1;
    const int L = taps - 1;
    const float* old = tail + (size_t)seq_slots[ch.seq] * (L > 0 ? L : 1) * conv_cols;
    // the input `back` tokens before token t of the chunk, t - back among the step's tokens or before them
    auto input = [&](int t, int c) {
        return ch.start + t >= 0 ? a[(size_t)(ch.first + t) * row_len + c] : old[(size_t)(L + ch.start + t) * conv_cols + c];
    };
    // (places of 64 x n values, 256 apart: no division in the loops)
    struct Walk {
        int t, j, dt, dj, n;
        __device__ Walk(int at, int n) : t(at / n), j(at % n), dt(256 / n), dj(256 % n), n(n) {}
        __device__ void step() {
            t += dt;
            j += dj;
            if (j >= n) {
                j -= n;
                ++t;
            }
        }
    };
    for (Walk at(tid, width); at.t < 4; at.step()) {
        const int ci = at.j, t0 = at.t * 16, c = c0 + ci;
        if (TAPS == 4) {
            const float4 w = *reinterpret_cast<const float4*>(conv_w + (size_t)c * 4);
            float x[19];
            if (t0 + 16 <= ch.count && ch.start + t0 >= 3) {
                const float* from = a + (size_t)(ch.first + t0 - 3) * row_len + c;
#pragma unroll
                for (int i = 0; i < 19; ++i, from += row_len) x[i] = *from;
            } else {
#pragma unroll
                for (int i = 0; i < 19; ++i) x[i] = t0 < ch.count && t0 + i - 3 < ch.count ? input(t0 + i - 3, c) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float acc = fmaf(w.x, x[i], 0.f);
                acc = fmaf(w.y, x[i + 1], acc);
                acc = fmaf(w.z, x[i + 2], acc);
                acc = fmaf(w.w, x[i + 3], acc);
                pack_y[(t0 + i) * ld + ci] = t0 + i < ch.count ? acc / (1.0f + expf(-acc)) : 0.f;
            }
        } else {
            for (int t = t0; t < t0 + 16; ++t) {
                float acc = 0.f;
                if (t < ch.count)
                    for (int j = 0; j < taps; ++j) acc = fmaf(conv_w[(size_t)c * taps + j], input(t - L + j, c), acc);
                pack_y[t * ld + ci] = acc / (1.0f + expf(-acc));
            }
        }
    }
    __syncthreads();
    if (!head) {
        float* to = values + ((size_t)blockIdx.x * H + (piece - 2 * G)) * kDC * vp;
        int it = tid;
        for (Walk at(tid, vp); at.t < kDC; at.step(), it += 256) to[it] = at.j < vdim ? pack_y[at.t * ld + at.j] : 0.f;
        return;
    }
    for (int t = warp; t < kDC; t += 8) {
        float ss = 0.f;
        for (int d = lane; d < dim; d += 32) ss = fmaf(pack_y[t * ld + d], pack_y[t * ld + d], ss);
        ss = warp_sum(ss);
        if (lane == 0) scale[t] = (piece < G ? q_scale : 1.0f) / sqrtf(ss + unit_eps);
    }
    __syncthreads();
    const int g = piece < G ? piece : piece - G;
    float* to = qk + ((size_t)blockIdx.x * G + g) * delta_qk_floats(dim) + (piece < G ? 0 : (size_t)kDC * dim);
    for (int it = tid; it < kDC * dim; it += 256) {
        const int t = it & (kDC - 1), d = it >> 6;
        to[it] = pack_y[t * ld + d] * scale[t];
    }
    if (piece < G) return;
    to += (size_t)kDC * dim;
    int it = tid;
    for (Walk at(tid, dim); at.t < kDC; at.step(), it += 256) to[it] = pack_y[at.t * ld + at.j] * scale[at.t];
}

// W [dim][64] (a row per value of the key) and U0 [64][vp].  128 threads, two columns each of the right sides
// [e^c beta k | beta v], whose 64 unknowns stay in registers: the substitution is one unrolled triangle.
template <int DIM>
__global__ void __launch_bounds__(128, 2)
delta_solve_kernel(const float* __restrict__ qk, const float* values, const float* __restrict__ beta,
                   const double* __restrict__ logs, float* __restrict__ w_out, float* u_out, int H, int G,
                   int vp) {
    extern __shared__ __align__(16) float solve_smem[];
    float* kt = solve_smem;         // [DIM][64]
    float* lower = kt + DIM * kDC;  // [64][64]: minus the system below its diagonal
    __shared__ double cs[kDC];
    __shared__ float bs[kDC], bg[kDC];
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, h = blockIdx.y, g = h / (H / G);
    const float* from = qk + ((size_t)blockIdx.x * G + g) * delta_qk_floats(DIM);
    const size_t unit = (size_t)blockIdx.x * H + h;
    for (int it = tid; it < DIM * kDC / 4; it += 128) copy16_or_zero(kt + it * 4, from + (size_t)kDC * DIM + it * 4, true);
    copy_commit();
    if (tid < kDC) {
        cs[tid] = logs[unit * kDC + tid];
        bs[tid] = beta[unit * kDC + tid];
        bg[tid] = bs[tid] * expf((float)cs[tid]);
    }
    copy_wait<0>();
    __syncthreads();
    {
        unsigned long long acc[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll 4
        for (int d = 0; d < DIM; ++d) {
            const float4 rl = load4(kt + d * kDC + ty * 8), rh = load4(kt + d * kDC + ty * 8 + 4);
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(kt + d * kDC + tx * 4);
            const float r[8] = {rl.x, rl.y, rl.z, rl.w, rh.x, rh.y, rh.z, rh.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long ri = both(r[i]);
                fma2(acc[i][0], ri, k.x);
                fma2(acc[i][1], ri, k.y);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int i = ty * 8 + r;
            const float2 a = halves(acc[r][0]), b = halves(acc[r][1]);
            const float x[4] = {a.x, a.y, b.x, b.y};
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = tx * 4 + e;
                y[e] = j < i ? -x[e] * (bs[i] * expf((float)(cs[i] - cs[j]))) : 0.f;
            }
            store4(lower + i * kDC + tx * 4, make_float4(y[0], y[1], y[2], y[3]));
        }
    }
    __syncthreads();
    const int cols = DIM + vp;
    for (int col = tid * 2; col < cols; col += 256) {  // (vp is a multiple of four: a pair lies in one right side)
        const bool is_w = col < DIM;
        const float* rhs = is_w ? from + (size_t)2 * kDC * DIM + col : values + unit * kDC * vp + (col - DIM);
        const int ld = is_w ? DIM : vp;
        const float* factor = is_w ? bg : bs;
        float x[kDC], y[kDC];
        constexpr int AHEAD = 8;  // rows of the right side fetched ahead
        float2 next[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) next[i] = *reinterpret_cast<const float2*>(rhs + (size_t)i * ld);
#pragma unroll
        for (int i = 0; i < kDC; ++i) {
            const float f = factor[i];
            float a = next[i % AHEAD].x * f, b = next[i % AHEAD].y * f;
            if (i + AHEAD < kDC) next[i % AHEAD] = *reinterpret_cast<const float2*>(rhs + (size_t)(i + AHEAD) * ld);
#pragma unroll
            for (int j4 = 0; j4 < (i + 3) / 4; ++j4) {
                const float4 l = load4(lower + i * kDC + j4 * 4);
                const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j4 * 4 + e < i) {
                        a = fmaf(lv[e], x[j4 * 4 + e], a);
                        b = fmaf(lv[e], y[j4 * 4 + e], b);
                    }
            }
            x[i] = a;
            y[i] = b;
        }
        if (is_w) {
            float* to = w_out + (unit * DIM + col) * kDC;
#pragma unroll
            for (int i = 0; i < kDC; i += 4) {
                store4(to + i, make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]));
                store4(to + kDC + i, make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]));
            }
        } else {
            float* to = u_out + unit * kDC * vp + (col - DIM);
#pragma unroll
            for (int i = 0; i < kDC; ++i) *reinterpret_cast<float2*>(to + (size_t)i * vp) = make_float2(x[i], y[i]);
        }
    }
}

// 256 threads, 32 columns of the state in shared memory from chunk to chunk.  Both products split their sum among the
// warps (8 x 8 outputs a thread) and meet in shared memory, in the order of the splits; while one multiplies, the other's
// operand of the next chunk is on its way.  U0 becomes U in place.
template <int DIM>
__global__ void __launch_bounds__(256)
delta_chain_kernel(const float* __restrict__ qk, const float* __restrict__ w, float* u, const double* __restrict__ logs,
                   float* __restrict__ before, float* __restrict__ state, const int* __restrict__ seq_slots,
                   const int* __restrict__ seq_count, const int* __restrict__ seq_first_chunk, int wave0, int wave_n, int H,
                   int G, int vdim, int vp) {
    constexpr int CW = 32, KW = DIM / 8;             // the state's rows per warp in the first product
    constexpr int SPLIT = DIM == 128 ? 4 : 8, KT = kDC / SPLIT;  // the tokens per split in the second
    extern __shared__ __align__(16) float chain_smem[];
    float* ws = chain_smem;             // [DIM][64]
    float* ks = ws + DIM * kDC;         // [64][DIM]
    float* u0s = ks + DIM * kDC;        // [64][32]
    float* us = u0s + kDC * CW;         // [64][32]: U times e^(c - c_j)
    float* ss = us + kDC * CW;          // [DIM][32]
    float* red = ss + DIM * CW;         // [8][64][32] or [SPLIT][DIM][32]
    __shared__ float left[2][kDC], whole[2];
    __shared__ int mine;
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, col0 = blockIdx.x * CW, g = h / (H / G), n_seqs = gridDim.z;
    // The longest sequences first: CTAs start in the order of their numbers, one to an SM, and a walk is serial (a prompt
    // of 2,048 tokens beside one of 555 in the order of the batch: 331 us, so 256).
    if (n_seqs <= 64) {
        if (tid < n_seqs) {
            const int n = seq_first_chunk[tid + 1] - seq_first_chunk[tid];
            int rank = 0;
            for (int s = 0; s < n_seqs; ++s) {
                const int m = seq_first_chunk[s + 1] - seq_first_chunk[s];
                rank += m > n || (m == n && s < tid);
            }
            if (rank == (int)blockIdx.z) mine = tid;
        }
    } else if (tid == 0) {
        mine = blockIdx.z;
    }
    __syncthreads();
    const int seq = mine;
    const int c0 = max(seq_first_chunk[seq], wave0), c1 = min(seq_first_chunk[seq + 1], wave0 + wave_n);  // among the wave's
    if (c1 <= c0) return;
    float* slot = state + ((size_t)seq_slots[seq] * H + h) * DIM * vdim;
    for (int it = tid; it < DIM * CW; it += 256) {
        const int d = it >> 5, j = col0 + (it & 31);
        ss[it] = j < vdim ? slot[(size_t)d * vdim + j] : 0.f;
    }
    auto bring_w = [&](int c) {  // and U0
        if (c < c1) {
            const size_t unit = (size_t)c * H + h;
            for (int it = tid; it < DIM * kDC / 4; it += 256) copy16_or_zero(ws + it * 4, w + unit * DIM * kDC + it * 4, true);
            for (int it = tid; it < kDC * CW / 4; it += 256) {
                const int t = it >> 3, j = col0 + (it & 7) * 4;
                copy16_or_zero(u0s + it * 4, u + unit * kDC * vp + (j < vp ? (size_t)t * vp + j : 0), j < vp);
            }
        }
        copy_commit();
    };
    auto bring_k = [&](int c) {
        if (c < c1) {
            const float* from = qk + ((size_t)c * G + g) * delta_qk_floats(DIM) + (size_t)2 * kDC * DIM;
            for (int it = tid; it < DIM * kDC / 4; it += 256) copy16_or_zero(ks + it * 4, from + it * 4, true);
        }
        copy_commit();
    };
    bring_w(c0);
    bring_k(c0);
    if (tid < kDC) {
        const double* lg = logs + ((size_t)c0 * H + h) * kDC;
        left[0][tid] = expf((float)(lg[kDC - 1] - lg[tid]));
        if (tid == 0) whole[0] = expf((float)lg[kDC - 1]);
    }
    for (int c = c0; c < c1; ++c) {
        const size_t unit = (size_t)c * H + h;
        const int now = (c - c0) & 1;
        copy_wait<1>();   // W and U0 (K may still be on its way)
        __syncthreads();  // ... and the state
        for (int it = tid; it < DIM * CW / 4; it += 256) {  // the state before the chunk
            const int d = it >> 3, j = col0 + (it & 7) * 4;
            if (j < vp) store4(before + unit * DIM * vp + (size_t)d * vp + j, load4(ss + it * 4));
        }
        {   // W S: warp w takes rows KW w .. of the state; lane (ty, tx): tokens 4 ty .. and 32 + 4 ty .., columns 4 tx .. and 16 + 4 tx ..
            const int tx = lane & 3, ty = lane >> 2;
            unsigned long long acc[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
            for (int k = warp * KW; k < warp * KW + KW; ++k) {
                const float4 al = load4(ws + k * kDC + ty * 4), ah = load4(ws + k * kDC + 32 + ty * 4);
                const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(ss + k * CW + tx * 4);
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(ss + k * CW + 16 + tx * 4);
                const float av[8] = {al.x, al.y, al.z, al.w, ah.x, ah.y, ah.z, ah.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned long long ai = both(av[i]);
                    fma2(acc[i][0], ai, b0.x);
                    fma2(acc[i][1], ai, b0.y);
                    fma2(acc[i][2], ai, b1.x);
                    fma2(acc[i][3], ai, b1.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float* to = red + ((warp * kDC) + (i < 4 ? 0 : 32) + ty * 4 + (i & 3)) * CW;
                *reinterpret_cast<ulonglong2*>(to + tx * 4) = make_ulonglong2(acc[i][0], acc[i][1]);
                *reinterpret_cast<ulonglong2*>(to + 16 + tx * 4) = make_ulonglong2(acc[i][2], acc[i][3]);
            }
        }
        __syncthreads();
        for (int it = tid; it < kDC * CW / 4; it += 256) {
            float4 x = load4(u0s + it * 4);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const float4 y = load4(red + s * kDC * CW + it * 4);
                x = make_float4(x.x - y.x, x.y - y.y, x.z - y.z, x.w - y.w);
            }
            const int t = it >> 3, j = col0 + (it & 7) * 4;
            if (j < vp) store4(u + unit * kDC * vp + (size_t)t * vp + j, x);
            const float f = left[now][t];
            store4(us + it * 4, make_float4(x.x * f, x.y * f, x.z * f, x.w * f));
        }
        copy_wait<0>();   // K
        __syncthreads();
        bring_w(c + 1);   // (W and U0 are done with)
        double log_end = 0.0, log_own = 0.0;  // the next chunk's, on their way under the product
        if (tid < kDC && c + 1 < c1) {
            const double* lg = logs + (unit + H) * kDC;
            log_end = lg[kDC - 1];
            log_own = lg[tid];
        }
        {   // K^T U: a split takes KT tokens; 8 rows and 8 columns of the state a thread
            constexpr int TPS = 256 / SPLIT;  // threads of a split: DIM / 8 x 4
            const int split = tid / TPS, t = tid % TPS, tx = t & 3, ty = t >> 2;
            unsigned long long acc[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
            for (int k = split * KT; k < split * KT + KT; ++k) {
                const float4 al = load4(ks + k * DIM + ty * 4), ah = load4(ks + k * DIM + DIM / 2 + ty * 4);
                const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(us + k * CW + tx * 4);
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(us + k * CW + 16 + tx * 4);
                const float av[8] = {al.x, al.y, al.z, al.w, ah.x, ah.y, ah.z, ah.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned long long ai = both(av[i]);
                    fma2(acc[i][0], ai, b0.x);
                    fma2(acc[i][1], ai, b0.y);
                    fma2(acc[i][2], ai, b1.x);
                    fma2(acc[i][3], ai, b1.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float* to = red + (split * DIM + (i < 4 ? 0 : DIM / 2) + ty * 4 + (i & 3)) * CW;
                *reinterpret_cast<ulonglong2*>(to + tx * 4) = make_ulonglong2(acc[i][0], acc[i][1]);
                *reinterpret_cast<ulonglong2*>(to + 16 + tx * 4) = make_ulonglong2(acc[i][2], acc[i][3]);
            }
        }
        if (tid < kDC) {
            left[now ^ 1][tid] = expf((float)(log_end - log_own));
            if (tid == 0) whole[now ^ 1] = expf((float)log_end);
        }
        __syncthreads();
        bring_k(c + 1);
        const float keep = whole[now];
        for (int it = tid; it < DIM * CW / 4; it += 256) {
            const float4 s = load4(ss + it * 4);
            float4 x = make_float4(s.x * keep, s.y * keep, s.z * keep, s.w * keep);
#pragma unroll
            for (int q = 0; q < SPLIT; ++q) {
                const float4 y = load4(red + q * DIM * CW + it * 4);
                x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
            }
            store4(ss + it * 4, x);
        }
        __syncthreads();  // the sums are read
    }
    copy_wait<0>();
    for (int it = tid; it < DIM * CW; it += 256) {
        const int d = it >> 5, j = col0 + (it & 31);
        if (j < vdim) slot[(size_t)d * vdim + j] = ss[it];
    }
}

template <int BV>
__global__ void __launch_bounds__(128, 3)
delta_read_kernel(const float* __restrict__ qk, const float* __restrict__ u, const double* __restrict__ logs,
                  const float* __restrict__ before, const int* __restrict__ chunks, const int* __restrict__ seq_first_row,
                  const int* __restrict__ seq_count, float* __restrict__ o_raw, int H, int G, int dim, int vdim, int vp) {
    extern __shared__ __align__(16) float read_smem[];
    __shared__ double cs[kDC];
    __shared__ float carry[kDC];
    pdl_wait();
    pdl_launch_dependents();
    const int h = blockIdx.y, v0 = blockIdx.z * BV, g = h / (H / G);
    const DeltaChunk ch = delta_chunk(chunks, seq_first_row, seq_count, blockIdx.x);
    const size_t unit = (size_t)blockIdx.x * H + h;
    if (threadIdx.x < kDC) {
        cs[threadIdx.x] = logs[unit * kDC + threadIdx.x];
        carry[threadIdx.x] = expf((float)cs[threadIdx.x]);
    }
    __syncthreads();
    const float* q = qk + ((size_t)blockIdx.x * G + g) * delta_qk_floats(dim);
    unsigned long long acc[8][BV / 32];
    chunk_read_tile<BV>(q, q + (size_t)kDC * dim, before + unit * dim * vp, u + unit * kDC * vp, dim, vp, v0, ch.count,
                        read_smem, acc, [&](int i, int j, float x) { return j <= i ? x * expf((float)(cs[i] - cs[j])) : 0.f; },
                        [&](int i) { return carry[i]; });
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const bool aligned = (vdim & 3) == 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int t = ty * 8 + r;
        if (t >= ch.count) continue;
        float* row = o_raw + ((size_t)(ch.first + t) * H + h) * vdim;
#pragma unroll
        for (int c = 0; c < BV / 64; ++c) {
            const int j = v0 + c * 64 + tx * 4;
            const float2 a = halves(acc[r][2 * c]), b = halves(acc[r][2 * c + 1]);
            if (aligned) {
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

template <typename K>
static cudaError_t most_shared(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace nnis

// a, conv_w, tail, a_log, dt_bias as for nnis_delta_prep (the tail is read; nnis_delta_conv_tail moves it on); dim 64 or
// 128; chunks int32 [n_chunks, 2] = (sequence, first token of the chunk among the step's), 64 tokens each, with
// seq_first_chunk [n_seqs + 1].  Float32 scratch, vp = vdim rounded up to a multiple of four: qk [wave, G, 192 dim],
// u [wave, H, 64, vp], w [wave, H, dim, 64], before [wave, H, dim, vp], beta [wave, H, 64]; double logs [wave, H, 64]
// (of n_chunks, if these are fewer): `wave` chunks are worked at a time.  o_raw float32 [n, H vdim].
NNIS_API int nnis_delta_prompt(const float* a, const float* conv_w, const float* tail, const float* a_log,
                               const float* dt_bias, float* state, const int* seq_slots, const int* seq_first_row,
                               const int* seq_count, const int* chunks, int n_chunks, const int* seq_first_chunk, int wave,
                               float* qk, float* u, float* w, float* before, float* beta, double* logs, float* o_raw,
                               int n_seqs, int H, int G, int dim, int vdim, int taps, float unit_eps, float q_scale,
                               cudaStream_t stream) {
    using namespace nnis;
    if (n_seqs <= 0 || n_chunks <= 0 || wave <= 0 || H <= 0 || G <= 0 || H % G || vdim <= 0 || taps < 1 || !(unit_eps > 0.f) || !a ||
        !conv_w || !tail || !a_log || !dt_bias || !state || !seq_slots || !seq_first_row || !seq_count || !chunks ||
        !seq_first_chunk || !qk || !u || !w || !before || !beta || !logs || !o_raw)
        return NNIS_ERR_ARGUMENT;
    if ((dim != 64 && dim != 128) || vdim > 512 || taps > 64 || 2 * G + H + 1 > 65535 || n_seqs > 65535) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)conv_w | (uintptr_t)qk | (uintptr_t)u | (uintptr_t)w | (uintptr_t)before | (uintptr_t)o_raw) % 16)
        return NNIS_ERR_ALIGNMENT;
    const int vp = (vdim + 3) & ~3, bv = vp > 64 ? 128 : 64, width = dim > vdim ? dim : vdim;
    const int pack_smem = kDC * (width + 1) * 4, solve_smem = (dim + kDC) * kDC * 4;
    const int chain_smem = (2 * dim * kDC + 2 * kDC * 32 + dim * 32 + 8 * kDC * 32) * 4;  // (4 x 128 = 8 x 64 rows of sums)
    const int read_smem = (bv == 128 ? chunk_read_floats<128>() : chunk_read_floats<64>()) * 4;
    auto pack = taps == 4 ? delta_pack_kernel<4> : delta_pack_kernel<0>;
    auto solve = dim == 128 ? delta_solve_kernel<128> : delta_solve_kernel<64>;
    auto chain = dim == 128 ? delta_chain_kernel<128> : delta_chain_kernel<64>;
    auto read = bv == 128 ? delta_read_kernel<128> : delta_read_kernel<64>;
    cudaError_t e = most_shared(pack, pack_smem);
    if (e == cudaSuccess) e = most_shared(solve, solve_smem);
    if (e == cudaSuccess) e = most_shared(chain, chain_smem);
    if (e == cudaSuccess) e = most_shared(read, read_smem);
    for (int c0 = 0; c0 < n_chunks && e == cudaSuccess; c0 += wave) {
        const int n = n_chunks - c0 < wave ? n_chunks - c0 : wave;
        const int* own = chunks + 2 * c0;
        e = launch_dependent(pack, dim3(n, 2 * G + H + 1), 256, pack_smem, stream, a, conv_w, tail, a_log, dt_bias, own,
                             seq_slots, seq_first_row, seq_count, qk, u, beta, logs, H, G, dim, vdim, vp, taps, unit_eps,
                             q_scale);
        // (values become U0 in place: a CTA of the solve reads a column of its own values before it writes it)
        if (e == cudaSuccess)
            e = launch_dependent(solve, dim3(n, H), 128, solve_smem, stream, (const float*)qk, (const float*)u,
                                 (const float*)beta, (const double*)logs, w, u, H, G, vp);
        // (the chain numbers the chunks of all waves, so its scratch begins where the first wave's would)
        const size_t gone = (size_t)c0 * H;
        if (e == cudaSuccess)
            e = launch_dependent(chain, dim3((vp + 31) / 32, H, n_seqs), 256, chain_smem, stream,
                                 (const float*)(qk - (size_t)c0 * G * delta_qk_floats(dim)),
                                 (const float*)(w - gone * dim * kDC), u - gone * kDC * vp, (const double*)(logs - gone * kDC),
                                 before - gone * dim * vp, state, seq_slots, seq_count, seq_first_chunk, c0, n, H, G, vdim, vp);
        if (e == cudaSuccess)
            e = launch_dependent(read, dim3(n, H, (vp + bv - 1) / bv), 128, read_smem, stream, (const float*)qk,
                                 (const float*)u, (const double*)logs, (const float*)before, own, seq_first_row, seq_count,
                                 o_raw, H, G, dim, vdim, vp);
    }
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
