// The gated delta rule (delta_rule.cu) over a prompt, 64 tokens at a time.  With c_i the sum of the log decays of a
// chunk up to token i, S_0 the state before the chunk and u_i what token i writes,
//     S_i = e^(c_i) S_0 + sum_(j<=i) e^(c_i - c_j) k_j u_j^T
//     u_i + sum_(j<i) beta_i e^(c_i - c_j) (k_i . k_j) u_j = beta_i (v_i - e^(c_i) S_0^T k_i)
//     o_i = e^(c_i) S_0^T q_i + sum_(j<=i) e^(c_i - c_j) (q_i . k_j) u_j
// so a chunk is a unit lower triangular system with two right sides, U = U0 - W S, and products:
//   delta_pack    convolution, silu, unit vectors, beta and c of every chunk, in octets of eight neighbouring places;
//   delta_solve   a CTA per (chunk, head), all side by side: q_i . k_j and k_i . k_j, the triangle's inverse T, W and U0;
//   delta_chain   a CTA per (sequence, head, 64 columns) walks the chunks: [q; W] S, U = U0 - W S, S <- e^c S + K^T (e^(c - c_j) U),
//                 and the outputs.
// More chunks than the scratch holds go through the kernels in waves, the slot's state from one to the next (the same
// bits: the state is float32 there too).
// Every product of matrices is six products of bfloat16 parts on the tensor cores, exact parts of float32 values, summed in
// float32 64 places at a time (split_parts.cuh); the triangle is inverted in float32, c is double (differences of sums of up to
// 64 logs keep float32's digits), a decay of zero counts as e^-200, which is zero in float32 and leaves the tokens after it
// exact.  Distance from 64 bits 1.7e-7 to 4.9e-7 of the outputs' norm where float32 sums on the CUDA cores had 2.1e-7 to 1.1e-6.
//
// Against the walk in runs with a transition matrix per run (delta_rule.cu, which other key sizes and short prompts
// keep): a token costs 2.2 dim vdim + 64 (dim + vdim) multiply-adds or so instead of 2.3 times three dim vdim, all but the chain side
// by side.
// Two prompts of 2,048 and 555 tokens, 32 heads over 16 key heads of 128 x 128, on a B200: with float32 multiply-adds, in four
// kernels (substitution, states, reads), 61 + 148 + 255 + 133 us; now pack 56, solve 109, chain 178.
#include "async_copy.cuh"
#include "common.cuh"
#include "split_parts.cuh"
#include "tcgen05_helpers.cuh"

namespace nnis {

constexpr int kDC = 64;
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

// A packed (chunk, key head), octets of eight neighbouring places of one token: queries [dim / 8][64][8], keys [dim / 8][64][8],
// and of eight neighbouring tokens: keys [64 / 8][dim][8]; and (chunk, head): values [vp / 8][64][8].
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
        for (int it = tid; it < kDC * vp / 8; it += 256) {
            const int t = it & (kDC - 1), j0 = (it >> 6) * 8;
            const float* from = pack_y + t * ld + j0;
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = j0 + e < vdim ? from[e] : 0.f;
            store8(to + it * 8, x);
        }
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
    for (int it = tid; it < kDC * dim / 8; it += 256) {
        const int t = it & (kDC - 1);
        const float* from = pack_y + t * ld + (it >> 6) * 8;
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = from[e] * scale[t];
        store8(to + it * 8, x);
    }
    if (piece < G) return;
    to += (size_t)kDC * dim;
    const int shift = dim == 128 ? 7 : 6;  // (dim is 64 or 128)
    for (int it = tid; it < kDC * dim / 8; it += 256) {
        const int d = it & (dim - 1), t0 = (it >> shift) * 8;
        const float* from = pack_y + t0 * ld + d;
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = from[e * ld] * scale[t0 + e];
        store8(to + it * 8, x);
    }
}

// The scores of a chunk: octets of keys, each from its first key's row on.
constexpr int kDeltaScores = 8 * 288;
__host__ __device__ __forceinline__ int delta_score(int octet, int i) {
    return 8 * (64 * octet - 4 * octet * (octet - 1)) + (i - 8 * octet) * 8;
}

// Shared memory of the solve: two blocks of 64 places of dim, three parts each, a part [64 queries | 64 keys] of 128-byte rows.
// Once the products q . k and k . k are made, the queries' tiles hold the rest: T beta's parts in the first block's, the
// triangle itself (float32) in two of the second's and what its inversion multiplies in the third; the values' parts replace
// the keys'.
constexpr uint32_t kDsTile = 64 * 128, kDsPart = 2 * kDsTile, kDsBlock = 3 * kDsPart, kDsSmem = 2 * kDsBlock + 1024;
constexpr int kDsThreads = 256;

struct DeltaSolveShared {
    uint64_t done[4];
    uint32_t tmem;
    volatile int abort_flag;
    double cs[kDC];
    float bs[kDC], bg[kDC];
};

// (i, j) of the triangle, by words of 16 bytes that neighbouring rows keep in different banks
__device__ __forceinline__ int delta_tri(int i, int j) { return (i >> 5) * (int)(kDsPart / 4) + (i & 31) * kDC + (j ^ ((i & 7) << 2)); }

// T = (1 + L)^-1 in place of -L, a unit lower triangle of 64, by 256 threads: the four triangles of 16 on its diagonal a column
// a thread, then twice the lower left square as T22 (-L21) T11.  Sums over m stop at the row's own place, so a row that
// holds no numbers is felt by the rows after it alone.  The entries of T are bounded by one (unit keys, beta at most one), so the
// inverse costs no digits against a substitution.
__device__ __forceinline__ void delta_invert(float* tri, float* mid) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp < 4) {
        const int r0 = warp * 16, c = lane & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float a = i == c ? 1.f : 0.f, b = 0.f;
#pragma unroll
            for (int m4 = 0; m4 < (i + 3) / 4; ++m4) {
                const float4 l = load4(tri + delta_tri(r0 + i, r0 + m4 * 4));
                const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int m = m4 * 4 + e;
                    if (m >= i) continue;
                    if (e & 1) b = m >= c ? fmaf(lv[e], x[m], b) : b;
                    else a = m >= c ? fmaf(lv[e], x[m], a) : a;
                }
            }
            x[i] = a + b;
        }
        __syncwarp();
        if (lane < 16)
#pragma unroll
            for (int i = 0; i < 16; ++i) tri[delta_tri(r0 + i, r0 + c)] = i >= c ? x[i] : 0.f;
    }
    __syncthreads();
    {
        const int pair = tid >> 7, i = (tid & 127) >> 3, j = (tid & 7) * 2, r0 = pair * 32 + 16, c0 = pair * 32;
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const float l = tri[delta_tri(r0 + i, c0 + m)];
            const float2 t = load2(tri + delta_tri(c0 + m, c0 + j));
            a = m >= j ? fmaf(l, t.x, a) : a;
            b = m >= j + 1 ? fmaf(l, t.y, b) : b;
        }
        store2(mid + pair * 512 + i * 16 + j, a, b);
        __syncthreads();
        a = b = 0.f;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const float t = tri[delta_tri(r0 + i, r0 + m)];
            const float2 y = load2(mid + pair * 512 + m * 16 + j);
            a = m <= i ? fmaf(t, y.x, a) : a;
            b = m <= i ? fmaf(t, y.y, b) : b;
        }
        store2(tri + delta_tri(r0 + i, c0 + j), a, b);
        __syncthreads();
    }
    const int i = tid >> 3, j = (tid & 7) * 4;
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
        const float l = tri[delta_tri(32 + i, m)];
        const float4 t = load4(tri + delta_tri(m, j));
        y.x = m >= j ? fmaf(l, t.x, y.x) : y.x;
        y.y = m >= j + 1 ? fmaf(l, t.y, y.y) : y.y;
        y.z = m >= j + 2 ? fmaf(l, t.z, y.z) : y.z;
        y.w = m >= j + 3 ? fmaf(l, t.w, y.w) : y.w;
    }
    store4(mid + i * 32 + j, y);
    __syncthreads();
    y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
        const float t = tri[delta_tri(32 + i, 32 + m)];
        const float4 z = load4(mid + m * 32 + j);
        if (m <= i) {
            y.x = fmaf(t, z.x, y.x);
            y.y = fmaf(t, z.y, y.y);
            y.z = fmaf(t, z.z, y.z);
            y.w = fmaf(t, z.w, y.w);
        }
    }
    store4(tri + delta_tri(32 + i, j), y);
    __syncthreads();
}

// A CTA per (chunk, head), two to an SM: the scores P, W and U0, and for the chain e^(c - c_j) and e^(c_j) in the place of the
// logs.  What is multiplied on the tensor cores: [q; k] k^T (128 x 64, a sum of 64 places at a time), k^T (T e^c beta)^T and
// v^T (T beta)^T (128 x 64 each).  Rows that no number comes out of are made again by multiply-adds over their own tokens.
template <int DIM>
__global__ void __launch_bounds__(kDsThreads, 2)
delta_solve_kernel(const float* __restrict__ qk, float* u, const float* __restrict__ beta, double* logs,
                   float* __restrict__ w_out, float* __restrict__ scores, int H, int G, int vp, int* __restrict__ status) {
    extern __shared__ unsigned char solve_smem[];
    __shared__ DeltaSolveShared sh;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(solve_smem) + 1023) & ~(uintptr_t)1023);
    constexpr int BLOCKS = DIM / 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), h = blockIdx.y, g = h / (H / G);
    const size_t unit = (size_t)blockIdx.x * H + h;
    float* tri = reinterpret_cast<float*>(base + kDsBlock);
    float* mid = reinterpret_cast<float*>(base + kDsBlock + 2 * kDsPart);
    pdl_wait();
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) mbar_init(&sh.done[i], 1);
        sh.abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&sh.tmem, 256);
    const float* q = qk + ((size_t)blockIdx.x * G + g) * delta_qk_floats(DIM);
    const float* k = q + (size_t)kDC * DIM;
    // rows of the queries and keys, eight values an item: token `it % 64`, places from 8 (it / 64 % (dim / 8))
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const float* from = half ? k : q;
        constexpr int ITEMS = kDC * DIM / 8 / kDsThreads;
        unsigned long long v[ITEMS][4];
#pragma unroll
        for (int e = 0; e < ITEMS; ++e) load8(from + (size_t)(e * kDsThreads + tid) * 8, v[e]);
#pragma unroll
        for (int e = 0; e < ITEMS; ++e) {
            const int it = e * kDsThreads + tid, t = it & (kDC - 1), o = it >> 6;
            store_parts(base + (o >> 3) * kDsBlock + half * kDsTile + t * 128 + (((o & 7) ^ (t & 7)) << 4), kDsPart, v[e]);
        }
    }
    if (tid < kDC) {
        const double c = logs[unit * kDC + tid];
        sh.cs[tid] = c;
        sh.bs[tid] = beta[unit * kDC + tid];
        sh.bg[tid] = sh.bs[tid] * expf((float)c);
    }
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();  // (the next kernel's CTAs may start, and wait: every CTA of this one has its tensor memory)
    const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem, 0);
    const int row = (warp & 3) * 32 + lane, cg = warp >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    int waits = 0;
    auto wait_done = [&] {
        ok = __all_sync(0xffffffffu, mbar_wait(&sh.done[waits & 3], (uint32_t)(waits >> 2) & 1u)) && ok;
        ++waits;
        tc_fence_after();
    };
    if (warp == 0) {
        constexpr uint32_t id = instr_desc(128, 64);
        const uint64_t da = smem_desc_k128(smem_addr(base)), db = smem_desc_k128(smem_addr(base) + kDsTile);
#pragma unroll 1
        for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    warp_mma(tmem + b * 64, desc_advance(da, b * kDsBlock + split_part_a(p) * kDsPart + s * 32),
                           desc_advance(db, b * kDsBlock + split_part_b(p) * kDsPart + s * 32), id, (p | s) != 0);
        warp_commit(&sh.done[0]);
    }
    if (tid < kDC) {  // (the logs are in shared memory)
        float* factors = reinterpret_cast<float*>(logs + unit * kDC);
        factors[tid] = expf((float)(sh.cs[kDC - 1] - sh.cs[tid]));
        factors[kDC + tid] = expf((float)sh.cs[tid]);
    }
    wait_done();
    {   // scores of the queries (rows 0 to 63), and the system's triangle of the keys (rows 64 to 127)
        float x[32];
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                uint32_t t[16];
                tmem_load16_issue(tmem + lanes + (uint32_t)(b * 64 + cg * 32 + c), t);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) x[c + e] = b ? x[c + e] + __uint_as_float(t[e]) : __uint_as_float(t[e]);
            }
        tc_fence_before();
        const int i = row & 63;
        const double ci = sh.cs[i];
        if (row < 64) {
            float* to = scores + unit * kDeltaScores;
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const int j8 = cg * 4 + o;
                if (i < j8 * 8) continue;
                float y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int j = j8 * 8 + e;
                    y[e] = j <= i ? x[o * 8 + e] * expf((float)(ci - sh.cs[j])) : 0.f;
                }
                store8(to + delta_score(j8, i), y);
            }
        } else {
            const float bi = sh.bs[i];
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
                float y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = cg * 32 + j4 * 4 + e;
                    y[e] = j < i ? -x[j4 * 4 + e] * (bi * expf((float)(ci - sh.cs[j]))) : 0.f;
                }
                store4(tri + delta_tri(i, cg * 32 + j4 * 4), make_float4(y[0], y[1], y[2], y[3]));
            }
        }
    }
    __syncthreads();
    delta_invert(tri, mid);
    // parts of T with its columns weighed
    auto keep_triangle = [&](const float* by) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int it = e * kDsThreads + tid, i = it & (kDC - 1), o = it >> 6;
            const float4 a = load4(tri + delta_tri(i, o * 8)), b = load4(tri + delta_tri(i, o * 8 + 4));
            float y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            unsigned long long v[4];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = o * 8 + j <= i ? y[j] * by[o * 8 + j] : 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = pair_of(y[2 * j], y[2 * j + 1]);
            store_parts(base + i * 128 + ((o ^ (i & 7)) << 4), kDsPart, v);
        }
    };
    auto hand_over = [&] {
        fence_async_shared();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    };
    // 128 columns of k or v (rows of the result) times the triangle's 64 rows (its columns)
    auto multiply = [&](uint32_t to, int bar) {
        if (warp == 0) {
            constexpr uint32_t id = instr_desc(128, 64) | (1u << 15);
            const uint64_t mn = smem_desc_mn128(smem_addr(base) + kDsTile);
            const uint64_t da = (mn & ~((uint64_t)0x3FFF << 16)) | (uint64_t)(kDsBlock >> 4) << 16;
            const uint64_t db = smem_desc_k128(smem_addr(base));
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    warp_mma(tmem + to, desc_advance(da, split_part_a(p) * kDsPart + s * 2048),
                           desc_advance(db, split_part_b(p) * kDsPart + s * 32), id, (p | s) != 0);
            warp_commit(&sh.done[bar & 3]);
        }
    };
    // what this thread's column `c` of `rows` (octets, [64][8] each) gives tokens cg 32 .. of the result
    auto collect = [&](uint32_t place, const float* rows, int c, bool there, const float* by, float* to) {
        float x[32];
#pragma unroll
        for (int e0 = 0; e0 < 32; e0 += 16) {
            uint32_t t[16];
            tmem_load16_issue(tmem + lanes + place + (uint32_t)(cg * 32 + e0), t);
            tmem_load_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e0 + e] = __uint_as_float(t[e]);
        }
        tc_fence_before();
        bool fine = true;
#pragma unroll
        for (int e = 0; e < 32; ++e) fine = fine && isfinite(x[e]);
        if (__syncthreads_or(there && !fine)) {
            const float* from = rows + (size_t)(c >> 3) * kDC * 8 + (c & 7);
            if (there && !fine) {
#pragma unroll
                for (int e = 0; e < 32; ++e) x[e] = 0.f;
#pragma unroll 1
                for (int j = 0; j < kDC; ++j) {
                    const float y = from[j * 8] * by[j];
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        if (j <= cg * 32 + e) x[e] = fmaf(tri[delta_tri(cg * 32 + e, j)], y, x[e]);
                }
            }
            __syncthreads();  // (two threads read a column that they may write in place)
        }
        if (!there) return;
        float* out = to + (size_t)(c >> 3) * kDC * 8 + (c & 7);
#pragma unroll
        for (int e = 0; e < 32; ++e) out[(cg * 32 + e) * 8] = x[e];
    };
    keep_triangle(sh.bg);
    hand_over();
    multiply(128, 1);
    float* values = u + unit * kDC * vp;
    const int tiles = (vp + 127) / 128;
    unsigned long long v[4][4];
    auto load_values = [&](int tile) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int o = tile * 16 + ((e * kDsThreads + tid) >> 6);
            if (o * 8 < vp) load8(values + ((size_t)o * kDC + (tid & (kDC - 1))) * 8, v[e]);
            else v[e][0] = v[e][1] = v[e][2] = v[e][3] = 0ull;
        }
    };
    load_values(0);
    wait_done();  // (the keys and the triangle's parts are done with)
    keep_triangle(sh.bs);
#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int it = e * kDsThreads + tid, t = it & (kDC - 1), o = it >> 6;
            store_parts(base + kDsTile + (o >> 3) * kDsBlock + t * 128 + (((o & 7) ^ (t & 7)) << 4), kDsPart, v[e]);
        }
        hand_over();
        multiply(192, 2 + tile);
        if (tile == 0) collect(128, k, row, row < DIM, sh.bg, w_out + unit * kDC * DIM);
        if (tile + 1 < tiles) load_values(tile + 1);
        wait_done();
        collect(192, values, tile * 128 + row, tile * 128 + row < vp, sh.bs, values);
    }
    if (!ok) sh.abort_flag = 1;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
    if (tid == 0 && sh.abort_flag && status) atomicExch(status, 3);
}

// Tensor memory of the chain, in columns: the parts of [q; W] and of the weighed keys (both the products' left sides), the sums
// of 64 places of [q; W] S each, and those of the scores times U.  What the keys add to the state takes the first sums' place.
template <int DIM>
struct DeltaChainPlaces {
    static constexpr uint32_t rows_part = DIM / 2, keys = 3 * rows_part, keys_part = kDC / 2, sums = keys + 3 * keys_part,
                              outs = sums + DIM, all = outs + 64;
    static_assert(all <= 512);
};
constexpr int kDtCols = 64, kDtWorkers = 16, kDtThreads = 32 * (1 + kDtWorkers);
constexpr uint32_t kDtPart = 64 * 128, kDtFactors = 2 * kDC * 4;  // bytes of a part of U or the scores; of a chunk's decays

// Shared memory of the chain: parts of S (64-column rows), of U and of the scores, then what the next step splits, as it lies
// in memory: a row of q and W, the keys, the scores, U0.
template <int DIM>
struct DeltaChainSmem {
    static constexpr uint32_t s_part = DIM * 128, u = 3 * s_part, p = u + 3 * kDtPart, rows = p + 3 * kDtPart,
                              keys = rows + 2 * kDC * DIM * 4, scores = keys + kDC * DIM * 4, u0 = scores + kDeltaScores * 4,
                              factors = u0 + kDC * kDtCols * 4, all = factors + 2 * kDtFactors + 1024;
};

struct DeltaChainShared {
    uint64_t state_in, u_in, sums_done, state_done, outs_done, rows_here, keys_here;
    uint32_t tmem;
    volatile int abort_flag, any_bad;
    int seq, bad[kDtCols];  // of every column the first token whose U is no number
};

// A CTA per (sequence, head, 64 columns) walks the chunks: one warp brings the operands and issues the products, sixteen hold the
// state, 16 values a thread (place `row` of the key, columns 16 cg ..), and split what is multiplied.  A step: [q; W] S; U = U0 - W S,
// split; K^T (e^(c - c_j) U) into the state, which is split for the next step, and P U beside it for the outputs.
// What bounds it: the two products that wait for each other, 1,445 + 722 cycles of the tensor cores at 64 columns, and the way of
// their sums through the threads to the next one's operand, twice a step.
template <int DIM>
__global__ void __launch_bounds__(kDtThreads, 1)
delta_chain_kernel(const float* __restrict__ qk, const float* __restrict__ w, const float* __restrict__ u0,
                   const float* __restrict__ scores, const double* __restrict__ logs, float* __restrict__ state,
                   const int* __restrict__ seq_slots, const int* __restrict__ seq_first_row, const int* __restrict__ seq_count,
                   const int* __restrict__ seq_first_chunk, float* __restrict__ o_raw, int wave0, int wave_n, int H, int G,
                   int vdim, int vp, int* __restrict__ status) {
    using At = DeltaChainPlaces<DIM>;
    using Smem = DeltaChainSmem<DIM>;
    extern __shared__ unsigned char chain_smem[];
    __shared__ DeltaChainShared sh;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(chain_smem) + 1023) & ~(uintptr_t)1023);
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int h = blockIdx.y, col0 = blockIdx.x * kDtCols, g = h / (H / G), n_seqs = gridDim.z;
    // The longest sequences first: CTAs start in the order of their numbers, one to an SM, and a walk is serial.
    if (n_seqs <= 64) {
        if (tid < n_seqs) {
            const int n = seq_first_chunk[tid + 1] - seq_first_chunk[tid];
            int rank = 0;
            for (int s = 0; s < n_seqs; ++s) {
                const int m = seq_first_chunk[s + 1] - seq_first_chunk[s];
                rank += m > n || (m == n && s < tid);
            }
            if (rank == (int)blockIdx.z) sh.seq = tid;
        }
    } else if (tid == 0) {
        sh.seq = blockIdx.z;
    }
    __syncthreads();
    const int seq = sh.seq, first_chunk = seq_first_chunk[seq];
    const int c0 = max(first_chunk, wave0), c1 = min(seq_first_chunk[seq + 1], wave0 + wave_n);  // among the wave's
    if (c1 <= c0) return;
    if (tid == 0) {
        mbar_init(&sh.state_in, kDtWorkers);
        mbar_init(&sh.u_in, kDtWorkers);
        mbar_init(&sh.sums_done, 1);
        mbar_init(&sh.state_done, 1);
        mbar_init(&sh.outs_done, 1);
        mbar_init(&sh.rows_here, 1);
        mbar_init(&sh.keys_here, 1);
        sh.abort_flag = sh.any_bad = 0;
        mbar_fence_init();
    }
    if (tid < kDtCols) sh.bad[tid] = 0x7fffffff;
    if (warp == 0) tmem_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem, 0);
    if (warp == 0) {
        constexpr uint32_t id = instr_desc(128, 64) | (1u << 16);
        const uint64_t ds = smem_desc_mn128(smem_addr(base)), du = smem_desc_mn128(smem_addr(base + Smem::u));
        const uint64_t dp = smem_desc_k128(smem_addr(base + Smem::p));
        const uint32_t u0_bytes = (uint32_t)min(kDtCols, vp - col0) * kDC * 4;
        auto bring_rows = [&](int c) {
            if (lane || c >= c1) return;
            mbar_expect_tx(&sh.rows_here, 2 * kDC * DIM * 4);
            bulk_load(base + Smem::rows, qk + ((size_t)c * G + g) * delta_qk_floats(DIM), kDC * DIM * 4, &sh.rows_here);
            bulk_load(base + Smem::rows + kDC * DIM * 4, w + ((size_t)c * H + h) * kDC * DIM, kDC * DIM * 4, &sh.rows_here);
        };
        auto bring_keys = [&](int c) {  // and the scores, U0 and the decays
            if (lane || c >= c1) return;
            const size_t unit = (size_t)c * H + h;
            mbar_expect_tx(&sh.keys_here, kDC * DIM * 4 + kDeltaScores * 4 + u0_bytes + kDtFactors);
            bulk_load(base + Smem::keys, qk + ((size_t)c * G + g) * delta_qk_floats(DIM) + (size_t)2 * kDC * DIM, kDC * DIM * 4, &sh.keys_here);
            bulk_load(base + Smem::u0, u0 + (unit * vp + col0) * kDC, u0_bytes, &sh.keys_here);
            bulk_load(base + Smem::scores, scores + unit * kDeltaScores, kDeltaScores * 4, &sh.keys_here);
            bulk_load(base + Smem::factors + (uint32_t)((c - c0) & 1) * kDtFactors, logs + unit * kDC, kDtFactors, &sh.keys_here);
        };
        bring_rows(c0);
        bring_keys(c0);
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar, parity) && !sh.abort_flag);
            tc_fence_after();
            return ok;
        };
        for (int c = c0; c < c1; ++c) {
            const uint32_t parity = (uint32_t)(c - c0) & 1u;
            if (!wait(&sh.state_in, parity)) break;
            bring_rows(c + 1);  // (this step's are in tensor memory)
#pragma unroll 1
            for (int b = 0; b < DIM / 64; ++b)
#pragma unroll
                for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        warp_mma_ts(tmem + At::sums + b * 64, tmem + split_part_a(p) * At::rows_part + b * 32 + s * 8,
                                    desc_advance(ds, b * 8192 + split_part_b(p) * Smem::s_part + s * 2048), id, (p | s) != 0);
            warp_commit(&sh.sums_done);
            if (!wait(&sh.u_in, parity)) break;
            bring_keys(c + 1);
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    warp_mma_ts(tmem + At::sums, tmem + At::keys + split_part_a(p) * At::keys_part + s * 8,
                                desc_advance(du, split_part_b(p) * kDtPart + s * 2048), id, (p | s) != 0);
            warp_commit(&sh.state_done);
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    warp_mma(tmem + At::outs, desc_advance(dp, split_part_a(p) * kDtPart + s * 32),
                             desc_advance(du, split_part_b(p) * kDtPart + s * 2048), id, (p | s) != 0);
            warp_commit(&sh.outs_done);
        }
        if (!ok) sh.abort_flag = 1;
        __syncwarp();
    } else {
        const int worker = warp - 1, cg = worker >> 2, row = (warp & 3) * 32 + lane, t = row & 63;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const bool writes = row >= 64;  // a token's row of W S; else of its query
        const int n_cols = vdim - col0 - cg * 16;
        bool ok = true;
        auto wait = [&](uint64_t* bar, int step) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar, (uint32_t)step & 1u) && ok && !sh.abort_flag);
            tc_fence_after();
            return ok;
        };
        float s[16], x[16];  // the state; U0 where the thread writes, q . S elsewhere
        float* slot = state + ((size_t)seq_slots[seq] * H + h) * DIM * vdim + (size_t)row * vdim + col0 + cg * 16;
#pragma unroll
        for (int e = 0; e < 16; ++e) s[e] = row < DIM && e < n_cols ? slot[e] : 0.f;
        auto keep16 = [&](unsigned char* to, int r, uint32_t part, const float (&y)[16]) {
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                unsigned long long v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = pair_of(y[o * 8 + 2 * e], y[o * 8 + 2 * e + 1]);
                store_parts(to + r * 128 + (((cg * 2 + o) ^ (r & 7)) << 4), part, v);
            }
        };
        auto shared_octet = [&](uint32_t at, unsigned long long (&v)[4]) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(base + at), b = *reinterpret_cast<const ulonglong2*>(base + at + 16);
            v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
        };
        constexpr int RO = DIM / 32;  // octets of its row of q or W that a thread splits
        auto keep_rows = [&] {
            unsigned long long v[RO][4];
#pragma unroll
            for (int o = 0; o < RO; ++o)
                shared_octet(Smem::rows + (writes ? kDC * DIM * 4 : 0) + (uint32_t)((cg * RO + o) * kDC + t) * 32, v[o]);
            uint32_t r[4 * RO];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
#pragma unroll
                for (int e = 0; e < 4 * RO; ++e) r[e] = p < 2 ? next_part(v[e >> 2][e & 3]) : last_part(v[e >> 2][e & 3]);
                tmem_store_issue(tmem + lanes + p * At::rows_part + cg * 4 * RO, r);
            }
        };
        const int pj = (worker * 32 + lane) >> 6, pi = (worker * 32 + lane) & 63;
        auto keep_keys = [&](int step) {  // weighed, and the scores
            const uint32_t factors = Smem::factors + (uint32_t)(step & 1) * kDtFactors;
            unsigned long long v[2][4];
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                if (row < DIM) {
                    unsigned long long f[4];
                    shared_octet(Smem::keys + (uint32_t)((cg * 2 + o) * DIM + row) * 32, v[o]);
                    shared_octet(factors + (uint32_t)(cg * 2 + o) * 32, f);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 y = halves(v[o][e]), z = halves(f[e]);
                        v[o][e] = pair_of(y.x * z.x, y.y * z.y);
                    }
                } else {
                    v[o][0] = v[o][1] = v[o][2] = v[o][3] = 0ull;
                }
            }
            uint32_t r[8];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
#pragma unroll
                for (int e = 0; e < 8; ++e) r[e] = p < 2 ? next_part(v[e >> 2][e & 3]) : last_part(v[e >> 2][e & 3]);
                tmem_store_issue(tmem + lanes + At::keys + p * At::keys_part + cg * 8, r);
            }
            if (pi >= pj * 8) shared_octet(Smem::scores + (uint32_t)delta_score(pj, pi) * 4, v[0]);
            else v[0][0] = v[0][1] = v[0][2] = v[0][3] = 0ull;
            store_parts(base + Smem::p + pi * 128 + ((pj ^ (pi & 7)) << 4), kDtPart, v[0]);
        };
        const bool wide = (vdim & 3) == 0;
        const int first_row = seq_first_row[seq], count = seq_count[seq];
        auto put_outs = [&](int c) {
            const int at = (c - first_chunk) * kDC + t;
            const float carry = *reinterpret_cast<const float*>(base + Smem::factors + (uint32_t)((c - c0) & 1) * kDtFactors + (kDC + t) * 4);
            uint32_t y[16];
            tmem_load16_issue(tmem + lanes + At::outs + (uint32_t)(cg * 16), y);
            tmem_load_wait();
            if (at >= count) return;
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = fmaf(x[e], carry, __uint_as_float(y[e]));
            if (sh.any_bad)
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (at >= sh.bad[cg * 16 + e]) x[e] = __int_as_float(0x7fc00000);
            float* to = o_raw + ((size_t)(first_row + at) * H + h) * vdim + col0 + cg * 16;
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
                if (wide) {
                    if (e < n_cols) store4(to + e, make_float4(x[e], x[e + 1], x[e + 2], x[e + 3]));
                } else {
#pragma unroll
                    for (int i = e; i < e + 4; ++i)
                        if (i < n_cols) to[i] = x[i];
                }
            }
        };
        auto hand_over = [&](uint64_t* bar) {
            fence_async_shared();
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        if (row < DIM) keep16(base, row, Smem::s_part, s);
        if (wait(&sh.rows_here, 0)) {
            keep_rows();
            hand_over(&sh.state_in);
        }
        for (int c = c0; ok && c < c1; ++c) {
            const int step = c - c0;
            const bool more = c + 1 < c1;
            // under [q; W] S: the outputs of the chunk before, this one's weighed keys and scores
            if (step > 0) {
                if (!wait(&sh.outs_done, step - 1)) break;
                if (!writes) put_outs(c - 1);
            }
            if (!wait(&sh.keys_here, step)) break;
            keep_keys(step);
            const float keep = *reinterpret_cast<const float*>(base + Smem::factors + (uint32_t)(step & 1) * kDtFactors + (2 * kDC - 1) * 4);
            if (writes) {
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
                    if (col0 + (cg * 2 + o) * 8 < vp) shared_octet(Smem::u0 + (uint32_t)((cg * 2 + o) * kDC + t) * 32, v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 y = halves(v[e]);
                        x[o * 8 + 2 * e] = y.x, x[o * 8 + 2 * e + 1] = y.y;
                    }
                }
            }
            if (!wait(&sh.sums_done, step)) break;
            {
                uint32_t y[16], z[16];
                tmem_load16_issue(tmem + lanes + At::sums + (uint32_t)(cg * 16), y);
                if (DIM > 64) tmem_load16_issue(tmem + lanes + At::sums + 64 + (uint32_t)(cg * 16), z);
                tmem_load_wait();
                float sum[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    sum[e] = DIM > 64 ? __uint_as_float(y[e]) + __uint_as_float(z[e]) : __uint_as_float(y[e]);
                if (writes) {
                    bool fine = true;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        x[e] -= sum[e];
                        fine = fine && isfinite(x[e]);
                    }
                    if (!fine) {  // earlier tokens' scores of it are zero, which a product of matrices would not leave out
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if (!isfinite(x[e])) {
                                atomicMin(&sh.bad[cg * 16 + e], (c - first_chunk) * kDC + t);
                                x[e] = 0.f;
                            }
                        sh.any_bad = 1;
                    }
                    keep16(base + Smem::u, t, kDtPart, x);
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) x[e] = sum[e];
                }
            }
            hand_over(&sh.u_in);
            if (more) {  // under the keys times U: the next step's rows
                if (!wait(&sh.rows_here, step + 1)) break;
                keep_rows();
            }
            if (!wait(&sh.state_done, step)) break;
            {
                uint32_t y[16];
                tmem_load16_issue(tmem + lanes + At::sums + (uint32_t)(cg * 16), y);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) s[e] = fmaf(s[e], keep, __uint_as_float(y[e]));
                if (sh.any_bad)
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if ((c - first_chunk + 1) * kDC > sh.bad[cg * 16 + e]) s[e] = __int_as_float(0x7fc00000);
            }
            if (more) {
                if (row < DIM) keep16(base, row, Smem::s_part, s);
                hand_over(&sh.state_in);
            }
        }
        if (ok && wait(&sh.outs_done, c1 - 1 - c0) && !writes) put_outs(c1 - 1);
        if (!ok) sh.abort_flag = 1;
        if (row < DIM)
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (e < n_cols) slot[e] = s[e];
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (tid == 0 && sh.abort_flag && status) atomicExch(status, 3);
}

template <typename K>
static cudaError_t most_shared(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace nnis

// a, conv_w, tail, a_log, dt_bias as for nnis_delta_prep (the tail is read; nnis_delta_conv_tail moves it on); dim 64 or
// 128; chunks int32 [n_chunks, 2] = (sequence, first token of the chunk among the step's), 64 tokens each, with
// seq_first_chunk [n_seqs + 1].  Float32 scratch on 32-byte boundaries, vp = vdim rounded up to a multiple of eight: qk [wave, G,
// 192 dim], u [wave, H, 64 vp], w [wave, H, 64 dim], scores [wave, H, 2304], beta [wave, H, 64]; double logs [wave, H, 64]
// (of n_chunks, if these are fewer): `wave` chunks are worked at a time.  o_raw float32 [n, H vdim].
NNIS_API int nnis_delta_prompt(const float* a, const float* conv_w, const float* tail, const float* a_log,
                               const float* dt_bias, float* state, const int* seq_slots, const int* seq_first_row,
                               const int* seq_count, const int* chunks, int n_chunks, const int* seq_first_chunk, int wave,
                               float* qk, float* u, float* w, float* scores, float* beta, double* logs, float* o_raw,
                               int n_seqs, int H, int G, int dim, int vdim, int taps, float unit_eps, float q_scale,
                               int* status, cudaStream_t stream) {
    using namespace nnis;
    if (n_seqs <= 0 || n_chunks <= 0 || wave <= 0 || H <= 0 || G <= 0 || H % G || vdim <= 0 || taps < 1 || !(unit_eps > 0.f) || !a ||
        !conv_w || !tail || !a_log || !dt_bias || !state || !seq_slots || !seq_first_row || !seq_count || !chunks ||
        !seq_first_chunk || !qk || !u || !w || !scores || !beta || !logs || !o_raw)
        return NNIS_ERR_ARGUMENT;
    if ((dim != 64 && dim != 128) || vdim > 512 || taps > 64 || 2 * G + H + 1 > 65535 || n_seqs > 65535) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)conv_w | (uintptr_t)o_raw) % 16 ||
        ((uintptr_t)qk | (uintptr_t)u | (uintptr_t)w | (uintptr_t)scores | (uintptr_t)logs) % 32)
        return NNIS_ERR_ALIGNMENT;
    const int vp = (vdim + 7) & ~7, width = dim > vdim ? dim : vdim;
    const int pack_smem = kDC * (width + 1) * 4;
    const int chain_smem = (int)(dim == 128 ? DeltaChainSmem<128>::all : DeltaChainSmem<64>::all);
    auto pack = taps == 4 ? delta_pack_kernel<4> : delta_pack_kernel<0>;
    auto solve = dim == 128 ? delta_solve_kernel<128> : delta_solve_kernel<64>;
    auto chain = dim == 128 ? delta_chain_kernel<128> : delta_chain_kernel<64>;
    cudaError_t e = most_shared(pack, pack_smem);
    if (e == cudaSuccess) e = most_shared(solve, (int)kDsSmem);
    if (e == cudaSuccess) e = most_shared(chain, chain_smem);
    for (int c0 = 0; c0 < n_chunks && e == cudaSuccess; c0 += wave) {
        const int n = n_chunks - c0 < wave ? n_chunks - c0 : wave;
        const int* own = chunks + 2 * c0;
        e = launch_dependent(pack, dim3(n, 2 * G + H + 1), 256, pack_smem, stream, a, conv_w, tail, a_log, dt_bias, own,
                             seq_slots, seq_first_row, seq_count, qk, u, beta, logs, H, G, dim, vdim, vp, taps, unit_eps,
                             q_scale);
        // (values become U0 in place, logs the decays that the chain takes: a CTA of the solve reads its own before it writes them)
        if (e == cudaSuccess)
            e = launch_dependent(solve, dim3(n, H), kDsThreads, kDsSmem, stream, (const float*)qk, u, (const float*)beta, logs,
                                 w, scores, H, G, vp, status);
        // (the chain numbers the chunks of all waves, so its scratch begins where the first wave's would)
        const size_t gone = (size_t)c0 * H;
        if (e == cudaSuccess)
            e = launch_dependent(chain, dim3((vdim + kDtCols - 1) / kDtCols, H, n_seqs), kDtThreads, chain_smem, stream,
                                 (const float*)(qk - (size_t)c0 * G * delta_qk_floats(dim)),
                                 (const float*)(w - gone * dim * kDC), (const float*)(u - gone * kDC * vp),
                                 (const float*)(scores - gone * kDeltaScores), (const double*)(logs - gone * kDC), state,
                                 seq_slots, seq_first_row, seq_count, seq_first_chunk, o_raw, c0, n, H, G, vdim, vp, status);
    }
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
