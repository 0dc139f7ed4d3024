// The gated delta rule (delta_rule.cu) over a prompt, 64 tokens at a time.  With c_i the sum of the log decays of a
// chunk up to token i, S_0 the state before the chunk and u_i what token i writes,
//     S_i = e^(c_i) S_0 + sum_(j<=i) e^(c_i - c_j) k_j u_j^T
//     u_i + sum_(j<i) beta_i e^(c_i - c_j) (k_i . k_j) u_j = beta_i (v_i - e^(c_i) S_0^T k_i)
//     o_i = e^(c_i) S_0^T q_i + sum_(j<=i) e^(c_i - c_j) (q_i . k_j) u_j
// so a chunk is a unit lower triangular system with two right sides, U = U0 - W S, and products:
//   delta_pack    convolution, silu, unit vectors, beta and c of every chunk, in the tiles that the products' operands come from;
//   delta_solve   a CTA per (chunk, head), all side by side: q_i . k_j and k_i . k_j, the triangle's inverse T, W and U0;
//   delta_chain   a CTA per (sequence, head, 64 columns) walks the chunks: [q; W] S, U = U0 - W S, S <- e^c S + K^T (e^(c - c_j) U),
//                 and the outputs.
// More chunks than the scratch holds go through the kernels in waves, the slot's state from one to the next (the same
// bits: the state is float32 there too).
// Every product of matrices is six products of bfloat16 parts on the tensor cores, exact parts of float32 values, summed in
// float32 in tensor memory over the 64 or 128 places of a chunk or a head (split_parts.cuh); the triangle is inverted in float32, c is
// double, then two floats (differences of sums of up to 64 logs keep float32's digits), a decay of zero counts as e^-200, which is
// zero in float32 and leaves the tokens after it exact.  Distance from 64 bits, independent keys to nearly parallel ones, of the outputs'
// norm 1.6e-7 to 5.2e-7 where float32 sums on the CUDA cores had 1.8e-7 to 1.1e-6, of the states' 0.9e-7 to 4.9e-7 (1.2e-7 to 1.0e-6).
//
// Against the walk in runs with a transition matrix per run (delta_rule.cu, which other key sizes and short prompts
// keep): a token costs 2.2 dim vdim + 64 (dim + vdim) multiply-adds or so instead of 2.3 times three dim vdim, all but the chain side
// by side.
// Two prompts of 2,048 and 555 tokens, 32 heads over 16 key heads of 128 x 128, on a B200: with float32 multiply-adds, in four
// kernels (substitution, states, reads), 61 + 148 + 255 + 133 us; now pack 57, solve 92, chain 128.
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

// Rows of a chunk in tiles of 32 columns, a row of 128 bytes a token with its 16-byte words swizzled: a warp that has a column a lane
// and one that has a row a lane both meet every bank once.  A packed (chunk, key head): queries and keys [dim / 32][64][32], keys
// with a row a place and a column a token [2][dim][32]; and (chunk, head): values, then U0 [vp / 32][64][32], W [dim / 32][64][32].
__host__ __device__ __forceinline__ int delta_at(int c, int t, int rows) {
    return ((c >> 5) * rows + t) * 32 + ((((c >> 2) & 7) ^ (t & 7)) << 2) + (c & 3);
}
__host__ __device__ __forceinline__ size_t delta_qk_floats(int dim) { return (size_t)3 * kDC * dim; }

// A CTA per (chunk, piece): q heads, k heads, value heads, and last the gates of all heads.  A thread walks 16 tokens of
// a channel; with TAPS (the taps when there are 4, else 0) the inputs before a token stay in registers.  Instructions bound it
// (104 a value with a division for each place and a test for each input, 79 us on the prompts above; 57 us now).
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
    // (four columns an item, eight neighbours to a row of a tile)
    auto put_rows = [&](float* to, int cols, int there, auto scale_of) {
        for (int it = tid; it < kDC * cols / 4; it += 256) {
            const int t = (it >> 3) & (kDC - 1), c = (it >> 9) * 32 + (((it ^ t) & 7) << 2);
            const float* from = pack_y + t * ld + c;
            const float f = scale_of(t);
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = c + e < there ? from[e] * f : 0.f;
            store4(to + it * 4, make_float4(x[0], x[1], x[2], x[3]));
        }
    };
    if (!head) {
        put_rows(values + ((size_t)blockIdx.x * H + (piece - 2 * G)) * kDC * vp, vp, vdim, [](int) { return 1.f; });
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
    put_rows(to, dim, dim, [&](int t) { return scale[t]; });
    if (piece < G) return;
    to += (size_t)kDC * dim;
    const int shift = dim == 128 ? 7 : 6;  // (dim is 64 or 128)
    for (int it = tid; it < kDC * dim / 4; it += 256) {
        const int d = (it >> 3) & (dim - 1), t = (it >> (3 + shift)) * 32 + (((it ^ d) & 7) << 2);
        const float* from = pack_y + t * ld + d;
        store4(to + it * 4, make_float4(from[0] * scale[t], from[ld] * scale[t + 1], from[2 * ld] * scale[t + 2], from[3 * ld] * scale[t + 3]));
    }
}

// The scores of a chunk: octets of keys, each from its first key's row on.
constexpr int kDeltaScores = 8 * 288;
__host__ __device__ __forceinline__ int delta_score(int octet, int i) {
    return 8 * (64 * octet - 4 * octet * (octet - 1)) + (i - 8 * octet) * 8;
}

// Shared memory of the solve: for every 64 places of dim three parts, each a tile of queries and one of keys (64 rows of 128
// bytes).  Once the products q . k and k . k are made, the queries' tiles hold the parts of T beta (first block), the triangle itself
// in float32 (two of the second's) and what its inversion multiplies (the third); the keys' first ones the parts of T beta e^c,
// the scores follow.
constexpr uint32_t kDsTile = 64 * 128, kDsPart = 2 * kDsTile, kDsBlock = 3 * kDsPart, kDsSmem = 2 * kDsBlock + kDeltaScores * 4 + 1024;
constexpr int kDsThreads = 512;

struct DeltaSolveShared {
    uint64_t done[2];  // in turn: a warp that still waits for one product is not overtaken by the next one's end
    uint32_t tmem;
    volatile int abort_flag;
    float ch[kDC], cl[kDC], bs[kDC], bg[kDC];  // the summed logs as two floats, beta, beta e^c
};

// (i, j) of the triangle, by words of 16 bytes that neighbouring rows keep in different banks
__device__ __forceinline__ int delta_tri(int i, int j) { return (i >> 5) * (int)(kDsPart / 4) + (i & 31) * kDC + (j ^ ((i & 7) << 2)); }

// T = (1 + L)^-1 in place of -L, a unit lower triangle of 64, by 512 threads: the four triangles of 16 on its diagonal a column
// a thread, then twice the lower left square as T22 (-L21) T11.  What a row gets comes from rows up to its own alone, also where
// they hold no numbers.  The entries of T are bounded by one (unit keys, beta at most one), so the inverse costs no digits
// against a substitution.
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
                    if (e & 1) b = fmaf(lv[e], x[m], b);
                    else a = fmaf(lv[e], x[m], a);
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
        const int pair = tid >> 8, i = (tid & 255) >> 4, j = tid & 15, r0 = pair * 32 + 16, c0 = pair * 32;
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int m = 0; m < 16; m += 4) {
            const float4 l = load4(tri + delta_tri(r0 + i, c0 + m));
            a = fmaf(l.x, tri[delta_tri(c0 + m, c0 + j)], a);
            b = fmaf(l.y, tri[delta_tri(c0 + m + 1, c0 + j)], b);
            a = fmaf(l.z, tri[delta_tri(c0 + m + 2, c0 + j)], a);
            b = fmaf(l.w, tri[delta_tri(c0 + m + 3, c0 + j)], b);
        }
        mid[pair * 256 + i * 16 + j] = a + b;
        __syncthreads();
        a = 0.f;
#pragma unroll
        for (int m = 0; m < 16; m += 4) {
            const float4 t = load4(tri + delta_tri(r0 + i, r0 + m));
            const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float y = mid[pair * 256 + (m + e) * 16 + j];
                a = m + e <= i ? fmaf(tv[e], y, a) : a;
            }
        }
        tri[delta_tri(r0 + i, c0 + j)] = a;
        __syncthreads();
    }
    // (32 x 32 outputs, 2 x 4 a thread: half the words of shared memory that 1 x 2 would read)
    const int i = (tid >> 3) * 2, j = (tid & 7) * 4;
    float y[2][4] = {};
    if (tid < 128) {
#pragma unroll
        for (int m = 0; m < 32; m += 4) {
            const float4 l0 = load4(tri + delta_tri(32 + i, m)), l1 = load4(tri + delta_tri(33 + i, m));
            const float a[4] = {l0.x, l0.y, l0.z, l0.w}, b[4] = {l1.x, l1.y, l1.z, l1.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 t = load4(tri + delta_tri(m + e, j));
                y[0][0] = fmaf(a[e], t.x, y[0][0]), y[0][1] = fmaf(a[e], t.y, y[0][1]), y[0][2] = fmaf(a[e], t.z, y[0][2]), y[0][3] = fmaf(a[e], t.w, y[0][3]);
                y[1][0] = fmaf(b[e], t.x, y[1][0]), y[1][1] = fmaf(b[e], t.y, y[1][1]), y[1][2] = fmaf(b[e], t.z, y[1][2]), y[1][3] = fmaf(b[e], t.w, y[1][3]);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) store4(mid + (i + r) * 32 + j, make_float4(y[r][0], y[r][1], y[r][2], y[r][3]));
    }
    __syncthreads();
    if (tid < 128) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) y[r][e] = 0.f;
#pragma unroll
        for (int m = 0; m < 32; m += 4) {
            const float4 t0 = load4(tri + delta_tri(32 + i, 32 + m)), t1 = load4(tri + delta_tri(33 + i, 32 + m));
            const float a[4] = {t0.x, t0.y, t0.z, t0.w}, b[4] = {t1.x, t1.y, t1.z, t1.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 z = load4(mid + (m + e) * 32 + j);
                if (m + e <= i) y[0][0] = fmaf(a[e], z.x, y[0][0]), y[0][1] = fmaf(a[e], z.y, y[0][1]), y[0][2] = fmaf(a[e], z.z, y[0][2]), y[0][3] = fmaf(a[e], z.w, y[0][3]);
                if (m + e <= i + 1) y[1][0] = fmaf(b[e], z.x, y[1][0]), y[1][1] = fmaf(b[e], z.y, y[1][1]), y[1][2] = fmaf(b[e], z.z, y[1][2]), y[1][3] = fmaf(b[e], z.w, y[1][3]);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) store4(tri + delta_tri(32 + i + r, j), make_float4(y[r][0], y[r][1], y[r][2], y[r][3]));
    }
    __syncthreads();
}

// A CTA per (chunk, head), two to an SM: the scores, W and U0, and for the chain e^(c_last - c_j) and e^(c_j) in the place of the
// logs.  On the tensor cores: [q; k] k^T (128 x 64, a sum of 64 places at a time), then columns of k and v (128, as the left side
// in tensor memory) times the 64 rows of a triangle.  A column that no number comes out of is made again by multiply-adds over
// each token's own past.
template <int DIM>
__global__ void __launch_bounds__(kDsThreads, 2)
delta_solve_kernel(const float* __restrict__ qk, float* u, const float* __restrict__ beta, double* logs,
                   float* __restrict__ w_out, float* __restrict__ scores, int H, int G, int vp, int* __restrict__ status) {
    extern __shared__ unsigned char solve_smem[];
    __shared__ DeltaSolveShared sh;
    unsigned char* base = shared_1024(solve_smem);
    constexpr int BLOCKS = DIM / 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), h = blockIdx.y, g = h / (H / G);
    const size_t unit = (size_t)blockIdx.x * H + h;
    float* tri = reinterpret_cast<float*>(base + kDsBlock);
    float* mid = reinterpret_cast<float*>(base + kDsBlock + 2 * kDsPart);
    float* own_scores = reinterpret_cast<float*>(base + 2 * kDsBlock);
    pdl_wait();
    if (tid == 0) {
        mbar_init(&sh.done[0], 1);
        mbar_init(&sh.done[1], 1);
        sh.abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&sh.tmem, 256);
    const float* q = qk + ((size_t)blockIdx.x * G + g) * delta_qk_floats(DIM);
    const float* k = q + (size_t)kDC * DIM;
    // rows of the queries and keys, eight values an item, eight neighbours to 64 places of a token
    {
        unsigned long long v[2 * BLOCKS][4];
        const int o = tid & 7, t = tid >> 3;
#pragma unroll
        for (int e = 0; e < 2 * BLOCKS; ++e) {
            const int b = e >> 1;
            load8((e & 1 ? k : q) + (size_t)((b * 2 + (o >> 2)) * kDC + t) * 32 + (((o & 3) * 2 ^ (t & 6)) << 2), v[e]);
        }
#pragma unroll
        for (int e = 0; e < 2 * BLOCKS; ++e) {
            if (t & 1) {  // (an octet's two words lie the other way round)
                const unsigned long long a = v[e][0], c = v[e][1];
                v[e][0] = v[e][2], v[e][1] = v[e][3], v[e][2] = a, v[e][3] = c;
            }
            store_parts(base + (e >> 1) * kDsBlock + (e & 1) * kDsTile + t * 128 + ((o ^ (t & 7)) << 4), kDsPart, v[e]);
        }
    }
    if (tid < kDC) {
        const double c = logs[unit * kDC + tid];
        const float b = beta[unit * kDC + tid];
        sh.ch[tid] = (float)c;
        sh.cl[tid] = (float)(c - (double)(float)c);
        sh.bs[tid] = b;
        sh.bg[tid] = b * expf((float)c);
    }
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();  // (the next kernel's CTAs may start, and wait: every CTA of this one has its tensor memory)
    const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem, 0);
    // this thread's column of k or v (with 16 tokens), or row of the scores (with 16 keys)
    const int row = (warp & 3) * 32 + lane, cg = warp >> 2, t0 = cg * 16;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    uint32_t made = 0, seen = 0;  // products
    auto wait_done = [&] {
        ok = __all_sync(0xffffffffu, mbar_wait(&sh.done[seen & 1u], (seen >> 1) & 1u)) && ok;
        ++seen;
        tc_fence_after();
    };
    auto hand_over = [&] {
        __syncwarp();
        fence_async_shared();
        tmem_store_wait();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    };
    // (what the first difference rounds off is added back, exact since the sums grow: one rounding of the logs' difference in all,
    // as with doubles; without it a decay is 4.4e-8 off at most instead of 2.2e-8)
    auto decay = [&](int i, int j) {
        const float hi = sh.ch[i], lo = sh.ch[j], d = hi - lo;
        return expf(d + (((hi - d) - lo) + (sh.cl[i] - sh.cl[j])));
    };
    auto collect = [&](uint32_t place, float (&x)[16]) {
        uint32_t y[16];
        tmem_load16_issue(tmem + lanes + place + (uint32_t)t0, y);
        tmem_load_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = __uint_as_float(y[e]);
    };
    // parts of this thread's 16 tokens of a column, at three places of tensor memory
    auto keep_left = [&](const float (&x)[16], uint32_t p0, uint32_t p1, uint32_t p2) {
        unsigned long long v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = pair_of(x[2 * e], x[2 * e + 1]);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            uint32_t r[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) r[e] = p < 2 ? next_part(v[e]) : last_part(v[e]);
            tmem_store_issue(tmem + lanes + (p == 0 ? p0 : p == 1 ? p1 : p2) + (uint32_t)cg * 8, r);
        }
    };
    // 128 columns, parts of 64 tokens at three places, times the 64 rows of a triangle
    auto multiply = [&](uint32_t to, uint32_t p0, uint32_t p1, uint32_t p2, const unsigned char* rows) {
        if (warp == 0) {
            constexpr uint32_t id = instr_desc(128, 64);
            const uint64_t db = smem_desc_k128(smem_addr(rows));
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const uint32_t a = split_part_a(p) == 0 ? p0 : split_part_a(p) == 1 ? p1 : p2;
                    warp_mma_ts(tmem + to, tmem + a + s * 8, desc_advance(db, split_part_b(p) * kDsPart + s * 32), id, (p | s) != 0);
                }
            warp_commit(&sh.done[made & 1u]);
        }
        ++made;
    };
    // what sums over tokens gave no number is made again, a token's own past alone
    auto mend = [&](float (&x)[16], bool there, const float* from, int c, const float* by) {
        bool fine = true;
#pragma unroll
        for (int e = 0; e < 16; ++e) fine = fine && isfinite(x[e]);
        tc_fence_before();
        const bool any = __syncthreads_or(there && !fine);
        tc_fence_after();
        if (!any) return;
        if (there && !fine) {
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = 0.f;
#pragma unroll 1
            for (int j = 0; j < t0 + 16; ++j) {
                const float y = from[delta_at(c, j, kDC)] * by[j];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (j <= t0 + e) x[e] = fmaf(tri[delta_tri(t0 + e, j)], y, x[e]);
            }
        }
        __syncthreads();  // (four threads read a column that they may write in place)
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
    ++made;
    float* values = u + unit * kDC * vp;
    float v[16];
    auto load_column = [&](const float* from, int c, bool there) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = there ? from[delta_at(c, t0 + e, kDC)] : 0.f;
    };
    // (columns of tensor memory: 0 to 127 q . k and k . k, then W and the values' first two parts; 128 to 223 the keys, then U0)
    load_column(k, row, row < DIM);
    keep_left(v, 128, 160, 192);
    if (tid < kDC) {  // (the logs are in shared memory)
        float* factors = reinterpret_cast<float*>(logs + unit * kDC);
        factors[tid] = decay(kDC - 1, tid);
        factors[kDC + tid] = expf(sh.ch[tid]);
    }
    load_column(values, row, row < vp);
    wait_done();
    __syncthreads();  // the queries' tiles are done with
    {
        float x[16];
        collect(0, x);
        if (BLOCKS > 1) {
            float y[16];
            collect(64, y);
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] += y[e];
        }
        const int i = row & 63;
        const bool before = (i | 31) < t0;  // (of the whole warp: its rows come before its keys)
        if (row < 64) {
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                if (i < t0 + o * 8) continue;
                float* to = own_scores + delta_score(cg * 2 + o, i);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int j = t0 + o * 8 + e;
                    x[o * 8 + e] = j <= i ? x[o * 8 + e] * decay(i, j) : 0.f;
                }
                store4(to, make_float4(x[o * 8], x[o * 8 + 1], x[o * 8 + 2], x[o * 8 + 3]));
                store4(to + 4, make_float4(x[o * 8 + 4], x[o * 8 + 5], x[o * 8 + 6], x[o * 8 + 7]));
            }
        } else {
            const float bi = sh.bs[i];
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
                float y[4] = {0.f, 0.f, 0.f, 0.f};
                if (!before)
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        const int j = t0 + e + f;
                        y[f] = j < i ? -x[e + f] * (bi * decay(i, j)) : 0.f;
                    }
                store4(tri + delta_tri(i, t0 + e), make_float4(y[0], y[1], y[2], y[3]));
            }
        }
    }
    hand_over();
    if (tid == 0) {  // (the scores leave as they lie)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(scores + unit * kDeltaScores),
                     "r"(smem_addr(own_scores)), "r"((uint32_t)(kDeltaScores * 4))
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    __syncwarp();  // (tensor memory is for whole warps)
    keep_left(v, 64, 96, 224);
    delta_invert(tri, mid);
    const int ti = tid & (kDC - 1), to8 = tid >> 6;  // an octet of the triangle's row
    auto keep_triangle = [&](unsigned char* to, const float* by) {
        const float4 a = load4(tri + delta_tri(ti, to8 * 8)), b = load4(tri + delta_tri(ti, to8 * 8 + 4));
        float y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        unsigned long long p[4];
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = to8 * 8 + j <= ti ? y[j] * by[to8 * 8 + j] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = pair_of(y[2 * j], y[2 * j + 1]);
        store_parts(to + ti * 128 + ((to8 ^ (ti & 7)) << 4), kDsPart, p);
    };
    keep_triangle(base + kDsTile, sh.bg);
    keep_triangle(base, sh.bs);
    hand_over();
    multiply(0, 128, 160, 192, base + kDsTile);
    wait_done();
    multiply(128, 64, 96, 224, base);
    float x[16];
    collect(0, x);
    mend(x, row < DIM, k, row, sh.bg);
    if (row < DIM)
#pragma unroll
        for (int e = 0; e < 16; ++e) w_out[unit * kDC * DIM + delta_at(row, t0 + e, kDC)] = x[e];
    const int tiles = (vp + 127) / 128;
#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
        const int c = tile * 128 + row;
        if (tile > 0) {
            keep_left(v, 64, 96, 224);
            hand_over();
            multiply(128, 64, 96, 224, base);
        }
        if (tile + 1 < tiles) load_column(values, c + 128, c + 128 < vp);
        wait_done();
        collect(128, x);
        mend(x, c < vp, values, c, sh.bs);
        if (c < vp)
#pragma unroll
            for (int e = 0; e < 16; ++e) values[delta_at(c, t0 + e, kDC)] = x[e];
    }
    if (!ok) sh.abort_flag = 1;
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
    if (tid == 0 && sh.abort_flag && status) atomicExch(status, 3);
}

// Tensor memory of the chain, in columns: the parts of [q; W], of the weighed keys and of the scores (the products' left sides),
// [q; W] S, whose place then takes what the keys add to the state, and the scores times U.
template <int DIM>
struct DeltaChainPlaces {
    static constexpr uint32_t rows_part = DIM / 2, keys = 3 * rows_part, keys_part = kDC / 2, scores = keys + 3 * keys_part,
                              sums = scores + 3 * keys_part, outs = sums + 64, all = outs + 64;
    static_assert(all <= 512);
};
constexpr int kDtCols = 64, kDtWorkers = 16, kDtThreads = 32 * (1 + kDtWorkers);
constexpr uint32_t kDtPart = 64 * 128, kDtFactors = 2 * kDC * 4;  // bytes of a part of U; of a chunk's decays

// Shared memory of the chain: parts of S (64-column rows) and of U, then what the next step splits, as it lies in memory: rows of q
// and W, the keys, U0, the scores, the decays of two steps; and a step's outputs on their way.
template <int DIM>
struct DeltaChainSmem {
    static constexpr uint32_t s_part = DIM * 128, u = 3 * s_part, rows = u + 3 * kDtPart, keys = rows + 2 * kDC * DIM * 4,
                              u0 = keys + kDC * DIM * 4, out = u0 + kDC * kDtCols * 4, scores = out + kDC * kDtCols * 4,
                              factors = scores + kDeltaScores * 4, all = factors + 2 * kDtFactors + 1024;
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
// What bounds it: the two products that wait for each other, 1,536 + 768 cycles of the tensor cores at 64 columns (1,700 and 1,100 to
// 1,500 beside the copies and splits that share shared memory with them), and the way of their sums through the threads to the
// next one's operand, 1,100 cycles each: 6,800 cycles a step.  Against a first form, 10,000 cycles a step: left sides in tensor memory
// instead of the scores in shared memory, rows of 128 swizzled bytes instead of octets, and outputs stored by TMA (row by row from
// the threads they held up the loads of shared memory of the other warps: 152 us of the kernel, 128 so).  Also tried: P W and P U0
// made by the solve so that the outputs are P U0 + (e^c q - P W) S: solve 161, chain 157.
template <int DIM>
__global__ void __launch_bounds__(kDtThreads, 1)
delta_chain_kernel(const __grid_constant__ CUtensorMap map_o, const float* __restrict__ qk, const float* __restrict__ w, const float* __restrict__ u0,
                   const float* __restrict__ scores, const double* __restrict__ logs, float* __restrict__ state,
                   const int* __restrict__ seq_slots, const int* __restrict__ seq_first_row, const int* __restrict__ seq_count,
                   const int* __restrict__ seq_first_chunk, float* __restrict__ o_raw, int wave0, int wave_n, int H, int G,
                   int vdim, int vp, int* __restrict__ status) {
    using At = DeltaChainPlaces<DIM>;
    using Smem = DeltaChainSmem<DIM>;
    extern __shared__ unsigned char chain_smem[];
    __shared__ DeltaChainShared sh;
    unsigned char* base = shared_1024(chain_smem);
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
#pragma unroll
            for (int p = 0; p < kSplitProducts; ++p)
#pragma unroll
                for (int s = 0; s < DIM / 16; ++s)
                    warp_mma_ts(tmem + At::sums, tmem + split_part_a(p) * At::rows_part + s * 8,
                                desc_advance(ds, split_part_b(p) * Smem::s_part + s * 2048), id, (p | s) != 0);
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
                    warp_mma_ts(tmem + At::outs, tmem + At::scores + split_part_a(p) * At::keys_part + s * 8,
                                desc_advance(du, split_part_b(p) * kDtPart + s * 2048), id, (p | s) != 0);
            warp_commit(&sh.outs_done);
        }
        if (!ok) sh.abort_flag = 1;
        __syncwarp();
    } else {
        const int worker = warp - 1, cg = worker >> 2, row = (warp & 3) * 32 + lane, t = row & 63;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const bool writes = (warp & 2) != 0;  // a token's row of W S; else of its query
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
        // four neighbouring places of a row of a tile (`word` of its eight)
        auto shared_word = [&](uint32_t tile, int r, int word) {
            return *reinterpret_cast<const ulonglong2*>(base + tile + (uint32_t)r * 128 + (uint32_t)((word ^ (r & 7)) << 4));
        };
        auto keep_left = [&](uint32_t at, uint32_t part, unsigned long long (&v)[8]) {
            uint32_t r[8];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
#pragma unroll
                for (int e = 0; e < 8; ++e) r[e] = p < 2 ? next_part(v[e]) : last_part(v[e]);
                tmem_store_issue(tmem + lanes + at + p * part, r);
            }
        };
        auto keep_rows = [&] {  // DIM / 4 places of its row of q or W
            const uint32_t from = Smem::rows + (writes ? kDC * DIM * 4 : 0);
#pragma unroll
            for (int i = 0; i < DIM / 64; ++i) {
                const int w0 = cg * (DIM / 16) + i * 4;
                unsigned long long v[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const ulonglong2 a = shared_word(from + (uint32_t)((w0 + e) >> 3) * 8192, t, (w0 + e) & 7);
                    v[2 * e] = a.x, v[2 * e + 1] = a.y;
                }
                keep_left(cg * (DIM / 8) + i * 8, At::rows_part, v);
            }
        };
        auto keep_keys = [&](int step) {  // weighed, and the scores
            const float* left = reinterpret_cast<const float*>(base + Smem::factors + (uint32_t)(step & 1) * kDtFactors) + cg * 16;
            unsigned long long v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (row < DIM) {
                    const ulonglong2 a = shared_word(Smem::keys + (uint32_t)((cg >> 1) * DIM) * 128, row, (cg & 1) * 4 + e);
                    const float2 x = halves(a.x), y = halves(a.y);
                    const float4 f = load4(left + e * 4);
                    v[2 * e] = pair_of(x.x * f.x, x.y * f.y), v[2 * e + 1] = pair_of(y.x * f.z, y.y * f.w);
                } else {
                    v[2 * e] = v[2 * e + 1] = 0ull;
                }
            }
            keep_left(At::keys + cg * 8, At::keys_part, v);
            if (writes) return;
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const ulonglong2* from = reinterpret_cast<const ulonglong2*>(base + Smem::scores + (uint32_t)delta_score(cg * 2 + o, max(t, (cg * 2 + o) * 8)) * 4);
                const bool there = t >= (cg * 2 + o) * 8;
                const ulonglong2 a = from[0], b = from[1];
                v[o * 4] = there ? a.x : 0ull, v[o * 4 + 1] = there ? a.y : 0ull;
                v[o * 4 + 2] = there ? b.x : 0ull, v[o * 4 + 3] = there ? b.y : 0ull;
            }
            keep_left(At::scores + cg * 8, At::keys_part, v);
        };
        const bool wide = (vdim & 3) == 0;
        const int worker_of_out = cg * 2 + (warp & 1);
        const int first_row = seq_first_row[seq], count = seq_count[seq];
        auto put_outs = [&](int c) {
            const int at = (c - first_chunk) * kDC + t;
            const float carry = *reinterpret_cast<const float*>(base + Smem::factors + (uint32_t)((c - c0) & 1) * kDtFactors + (kDC + t) * 4);
            uint32_t y[16];
            tmem_load16_issue(tmem + lanes + At::outs + (uint32_t)(cg * 16), y);
            tmem_load_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = fmaf(x[e], carry, __uint_as_float(y[e]));
            if (sh.any_bad)
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (at >= sh.bad[cg * 16 + e]) x[e] = __int_as_float(0x7fc00000);
            if (wide && n_cols >= 16 && (c - first_chunk) * kDC + (t | 31) < count) {  // the warp's 32 rows of 64 bytes, as one store
                unsigned char* mine = base + Smem::out + (uint32_t)(worker_of_out * 2048);
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    store4(reinterpret_cast<float*>(mine + lane * 64 + ((e ^ ((lane >> 1) & 3)) << 4)),
                           make_float4(x[e * 4], x[e * 4 + 1], x[e * 4 + 2], x[e * 4 + 3]));
                fence_async_shared();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&map_o, h * vdim + col0 + cg * 16, first_row + (c - first_chunk) * kDC + (t & 32), mine);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else if (at < count) {
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
            }
        };
        auto hand_over = [&](uint64_t* bar) {
            __syncwarp();
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
                for (int e = 0; e < 4; ++e) {
                    ulonglong2 a = make_ulonglong2(0ull, 0ull);
                    if (col0 + cg * 16 < vp) a = shared_word(Smem::u0 + (uint32_t)(cg >> 1) * 8192, t, (cg & 1) * 4 + e);
                    const float2 y = halves(a.x), z = halves(a.y);
                    x[e * 4] = y.x, x[e * 4 + 1] = y.y, x[e * 4 + 2] = z.x, x[e * 4 + 3] = z.y;
                }
            }
            if (!wait(&sh.sums_done, step)) break;
            {
                uint32_t y[16];
                tmem_load16_issue(tmem + lanes + At::sums + (uint32_t)(cg * 16), y);
                tmem_load_wait();
                float sum[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[e] = __uint_as_float(y[e]);
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
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
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

// Rows of the outputs for stores of 32 rows x 16 columns, 64 bytes a row, swizzled by fours of words.
static bool delta_out_map(CUtensorMap* map, float* o_raw, int rows, int cols) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 4};
    const cuuint32_t box[2] = {16, 32}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, o_raw, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
static cudaError_t most_shared(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace nnis

// a, conv_w, tail, a_log, dt_bias as for nnis_delta_prep (the tail is read; nnis_delta_conv_tail moves it on); dim 64 or
// 128; chunks int32 [n_chunks, 2] = (sequence, first token of the chunk among the step's), 64 tokens each, with
// seq_first_chunk [n_seqs + 1].  Float32 scratch on 32-byte boundaries, vp = vdim rounded up to a multiple of 32: qk [wave, G,
// 192 dim], u [wave, H, 64 vp], w [wave, H, 64 dim], scores [wave, H, 2304], beta [wave, H, 64]; double logs [wave, H, 64]
// (of n_chunks, if these are fewer): `wave` chunks are worked at a time.  o_raw float32 [n, H vdim].
NNIS_API int nnis_delta_prompt(const float* a, const float* conv_w, const float* tail, const float* a_log,
                               const float* dt_bias, float* state, const int* seq_slots, const int* seq_first_row,
                               const int* seq_count, const int* chunks, int n_chunks, const int* seq_first_chunk, int wave,
                               float* qk, float* u, float* w, float* scores, float* beta, double* logs, float* o_raw,
                               int n_seqs, int H, int G, int dim, int vdim, int taps, float unit_eps, float q_scale,
                               int n, int* status, cudaStream_t stream) {
    using namespace nnis;
    if (n <= 0 || n_seqs <= 0 || n_chunks <= 0 || wave <= 0 || H <= 0 || G <= 0 || H % G || vdim <= 0 || taps < 1 || !(unit_eps > 0.f) || !a ||
        !conv_w || !tail || !a_log || !dt_bias || !state || !seq_slots || !seq_first_row || !seq_count || !chunks ||
        !seq_first_chunk || !qk || !u || !w || !scores || !beta || !logs || !o_raw)
        return NNIS_ERR_ARGUMENT;
    if ((dim != 64 && dim != 128) || vdim > 512 || taps > 64 || 2 * G + H + 1 > 65535 || n_seqs > 65535) return NNIS_ERR_UNSUPPORTED;
    if (((uintptr_t)conv_w | (uintptr_t)o_raw) % 16 ||
        ((uintptr_t)qk | (uintptr_t)u | (uintptr_t)w | (uintptr_t)scores | (uintptr_t)logs) % 32)
        return NNIS_ERR_ALIGNMENT;
    const int vp = (vdim + 31) & ~31, width = dim > vdim ? dim : vdim;
    const int pack_smem = kDC * (width + 1) * 4;
    const int chain_smem = (int)(dim == 128 ? DeltaChainSmem<128>::all : DeltaChainSmem<64>::all);
    auto pack = taps == 4 ? delta_pack_kernel<4> : delta_pack_kernel<0>;
    auto solve = dim == 128 ? delta_solve_kernel<128> : delta_solve_kernel<64>;
    auto chain = dim == 128 ? delta_chain_kernel<128> : delta_chain_kernel<64>;
    cudaError_t e = most_shared(pack, pack_smem);
    if (e == cudaSuccess) e = most_shared(solve, (int)kDsSmem);
    if (e == cudaSuccess) e = most_shared(chain, chain_smem);
    CUtensorMap map_o = {};
    if (vdim % 4 == 0 && !delta_out_map(&map_o, o_raw, n, H * vdim)) return NNIS_ERR_UNSUPPORTED;
    for (int c0 = 0; c0 < n_chunks && e == cudaSuccess; c0 += wave) {
        const int n_own = n_chunks - c0 < wave ? n_chunks - c0 : wave;
        const int* own = chunks + 2 * c0;
        e = launch_dependent(pack, dim3(n_own, 2 * G + H + 1), 256, pack_smem, stream, a, conv_w, tail, a_log, dt_bias, own,
                             seq_slots, seq_first_row, seq_count, qk, u, beta, logs, H, G, dim, vdim, vp, taps, unit_eps,
                             q_scale);
        // (values become U0 in place, logs the decays that the chain takes: a CTA of the solve reads its own before it writes them)
        if (e == cudaSuccess)
            e = launch_dependent(solve, dim3(n_own, H), kDsThreads, kDsSmem, stream, (const float*)qk, u, (const float*)beta, logs,
                                 w, scores, H, G, vp, status);
        // (the chain numbers the chunks of all waves, so its scratch begins where the first wave's would)
        const size_t gone = (size_t)c0 * H;
        if (e == cudaSuccess)
            e = launch_dependent(chain, dim3((vdim + kDtCols - 1) / kDtCols, H, n_seqs), kDtThreads, chain_smem, stream, map_o,
                                 (const float*)(qk - (size_t)c0 * G * delta_qk_floats(dim)),
                                 (const float*)(w - gone * dim * kDC), (const float*)(u - gone * kDC * vp),
                                 (const float*)(scores - gone * kDeltaScores), (const double*)(logs - gone * kDC), state,
                                 seq_slots, seq_first_row, seq_count, seq_first_chunk, o_raw, c0, n_own, H, G, vdim, vp, status);
    }
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
