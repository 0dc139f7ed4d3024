// Row-wise kernels around the matrix products: embedding gather, RMSNorm,
// the gated activation, and RoPE fused with the store into the paged cache.
// The residual stream is float32 in both engine dtypes; T is the dtype of the
// matrix-product operands (float or bfloat16).  Statistics, angles and the
// activation are computed in float32 and rounded once on the store.
#include "async_copy.cuh"
#include "common.cuh"
#include "row_quads.cuh"

#include <stdlib.h>
#include <string.h>

namespace nnis {

bool dependent_launches() {
    static const bool on = [] {
        const char* v = getenv("NNIS_PDL");
        return !(v && strcmp(v, "0") == 0);
    }();
    return on;
}

// ---------------------------------------------------------------------------
// hidden[n, :] = table[token[n], :]  (widened exactly to float32)
// NNIS: crates/nnis-kernels/src/gather.rs:17-33.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void embed_kernel(const T* __restrict__ table, const int* __restrict__ tokens,
                             float* __restrict__ hidden, int n_tokens, int width, int vocab,
                             int* __restrict__ status, float scale) {
    int n = blockIdx.x;
    int token = tokens[n];
    bool bad = token < 0 || token >= vocab;
    if (bad) {
        if (threadIdx.x == 0) atomicExch(status, 1);
        token = 0;
    }
    const T* row = table + (size_t)token * width;
    float* out = hidden + (size_t)n * width;
    for (int i = threadIdx.x; i < width; i += blockDim.x) out[i] = bad ? 0.f : to_float(row[i]) * scale;
}

// The same, four neighbours a load (rows of a multiple of four values).
template <typename T>
__global__ void __launch_bounds__(256)
embed_quads_kernel(const T* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ hidden, int n_quads,
                   int vocab, int* __restrict__ status, float scale) {
    const int n = blockIdx.x, token = tokens[n];
    const bool bad = token < 0 || token >= vocab;
    if (bad && threadIdx.x == 0) atomicExch(status, 1);
    const T* row = table + (size_t)(bad ? 0 : token) * n_quads * 4;
    float* out = hidden + (size_t)n * n_quads * 4;
    for (int i = threadIdx.x; i < n_quads; i += 256) {
        const float4 v = load4(row + 4 * i);
        store4(out + 4 * i, bad ? make_float4(0.f, 0.f, 0.f, 0.f)
                                : make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale));
    }
}

// ---------------------------------------------------------------------------
// y = (x * 1/sqrt(mean(x^2) + eps)) * w, one block per output row; `rows`
// (optional) picks the input row of each output row.
// NNIS: crates/nnis-model/src/kernels.rs:15-48.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const int* __restrict__ rows,
                               const float* __restrict__ w, T* __restrict__ y, int width,
                               float eps) {
    __shared__ float partial[32];
    __shared__ float scale_s;
    // launched as a programmatic dependent: x comes from the kernel before this one
    pdl_wait();
    pdl_launch_dependents();
    int r = blockIdx.x;
    const float* in = x + (size_t)(rows ? rows[r] : r) * width;
    float ss = 0.f;
    for (int i = threadIdx.x; i < width; i += blockDim.x) ss = fmaf(in[i], in[i], ss);
    ss = warp_sum(ss);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    if (lane == 0) partial[warp] = ss;
    __syncthreads();
    if (warp == 0) {
        float v = lane < n_warps ? partial[lane] : 0.f;
        v = warp_sum(v);
        if (lane == 0) scale_s = 1.0f / sqrtf(v * (1.0f / (float)width) + eps);
    }
    __syncthreads();
    float s = scale_s;
    T* out = y + (size_t)r * width;
    for (int i = threadIdx.x; i < width; i += blockDim.x) out[i] = from_float<T>((in[i] * s) * w[i]);
}

// The same for rows of a multiple of four values, at most 1,024 Q: a CTA of 256 threads a row, the row and the weights in
// registers.  1,850 rows of 2,048: 10.5 -> 3.7 us on a B200 (23 MB, most of it from L2).
template <typename T, int Q>
__global__ void __launch_bounds__(256)
rmsnorm_quads_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ w,
                     T* __restrict__ y, int width, float eps) {
    __shared__ float partial[8];
    const int tid = threadIdx.x, n4 = width >> 2, r = blockIdx.x;
    float4 g[Q], v[Q];
#pragma unroll
    for (int j = 0; j < Q; ++j) g[j] = tid + 256 * j < n4 ? load4(w + 4 * (tid + 256 * j)) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();  // (the weights depend on no kernel)
    pdl_launch_dependents();
    const float* in = x + (size_t)(rows ? rows[r] : r) * width;
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < Q; ++j) {
        v[j] = tid + 256 * j < n4 ? load4(in + 4 * (tid + 256 * j)) : make_float4(0.f, 0.f, 0.f, 0.f);
        ss = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, ss))));
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) partial[tid >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) total += partial[k];
    const float s = 1.0f / sqrtf(total * (1.0f / (float)width) + eps);
    T* out = y + (size_t)r * width;
#pragma unroll
    for (int j = 0; j < Q; ++j)
        if (tid + 256 * j < n4)
            store4(out + 4 * (tid + 256 * j), make_float4((v[j].x * s) * g[j].x, (v[j].y * s) * g[j].y,
                                                          (v[j].z * s) * g[j].z, (v[j].w * s) * g[j].w));
}

// The same for many rows of moderate width (a multiple of 4, at most 1,024): a
// warp per row, the row kept in registers between the sum and the scaling, no
// barrier; eight rows per CTA.
template <typename T>
__global__ void __launch_bounds__(256)
rmsnorm_rows_kernel(const float* __restrict__ x, const int* __restrict__ rows,
                    const float* __restrict__ w, T* __restrict__ y, int n_rows, int width, float eps,
                    unsigned long long* trace) {
    trace_mark(trace, 0);
    const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
    const float4* w4 = reinterpret_cast<const float4*>(w);
    const int n4 = width >> 2;
    // the norm's weights depend on no kernel: they are fetched before the wait
    float4 g[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        int c = lane + 32 * j;
        g[j] = c < n4 ? w4[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    pdl_launch_dependents();
    trace_mark(trace, 2);
    trace_mark(trace, 3);
    if (r >= n_rows) {
        trace_mark(trace, 1);
        return;
    }
    const float4* in = reinterpret_cast<const float4*>(x + (size_t)(rows ? rows[r] : r) * width);
    float4 v[8];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        int c = lane + 32 * j;
        v[j] = c < n4 ? in[c] : make_float4(0.f, 0.f, 0.f, 0.f);
        ss = fmaf(v[j].x, v[j].x, ss);
        ss = fmaf(v[j].y, v[j].y, ss);
        ss = fmaf(v[j].z, v[j].z, ss);
        ss = fmaf(v[j].w, v[j].w, ss);
    }
    ss = warp_sum(ss);
    const float s = 1.0f / sqrtf(ss * (1.0f / (float)width) + eps);
    T* out = y + (size_t)r * width;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        int c = lane + 32 * j;
        if (c < n4)
            store4(out + c * 4, make_float4((v[j].x * s) * g[j].x, (v[j].y * s) * g[j].y, (v[j].z * s) * g[j].z,
                                            (v[j].w * s) * g[j].w));
    }
    trace_mark(trace, 1);
}

// ---------------------------------------------------------------------------
// out[n, i] = act(g[n, i]) * u[n, i], act silu or gelu's tanh form; gate and up are the two halves of one
// float32 row [2 * inter].  NNIS: crates/nnis-model/src/fused_swiglu.rs:14-27.
// ---------------------------------------------------------------------------
template <typename T, bool GELU>
__global__ void gate_mul_kernel(const float* __restrict__ gate_up, T* __restrict__ out,
                                size_t n_rows, int inter) {
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_rows * (size_t)inter) return;
    size_t n = idx / inter;
    int i = (int)(idx - n * inter);
    float g = gate_up[n * 2 * inter + i];
    float u = gate_up[n * 2 * inter + inter + i];
    const float act = GELU ? 0.5f * g * (1.0f + tanhf(0.79788456080286536f * (g + 0.044715f * g * g * g)))
                           : g / (1.0f + expf(-g));
    out[idx] = from_float<T>(act * u);
}

// ---------------------------------------------------------------------------
// Rotate-half RoPE on the q and k heads of a packed [n, (nq + 2 nkv) * d] row,
// in place, and store rotated k and plain v at each token's position of the
// paged cache.  cos/sin: [max_positions, d/2] float32.  With `rotate == 0` only
// the store happens; with nkv == 0 only q is rotated (a layer that reads another
// layer's cache).
// NNIS: crates/nnis-model/src/runtime_kernels.rs:38-66 and the append in
// crates/nnis-rt/src/kv_cache.rs:212-366.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void rope_store_kernel(T* __restrict__ qkv, const int* __restrict__ token_pos,
                                  const int* __restrict__ token_seq,
                                  const int* __restrict__ page_table, int table_cols,
                                  const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                  T* __restrict__ k_cache, T* __restrict__ v_cache, int nq, int nkv,
                                  int d, int page_size, int rotate) {
    int n = blockIdx.x;
    int pos = token_pos[n];
    if (pos < 0) return;  // a padding row: nothing to rotate, nothing to store
    int half = d >> 1;
    T* row = qkv + (size_t)n * (nq + 2 * nkv) * d;
    size_t page_base = 0;
    int in_page = 0;
    if (nkv > 0) {
        int page = page_table[(size_t)token_seq[n] * table_cols + pos / page_size];
        page_base = (size_t)page * nkv * page_size * d;
        in_page = pos % page_size;
    }
    int rot_items = (nq + nkv) * half;
    for (int it = threadIdx.x; it < rot_items; it += blockDim.x) {
        int head = it / half, j = it - head * half;
        T* h = row + (size_t)head * d;
        float a = to_float(h[j]), b = to_float(h[j + half]);
        float ra = a, rb = b;
        if (rotate) {
            float c = cos_t[(size_t)pos * half + j], s = sin_t[(size_t)pos * half + j];
            ra = a * c - b * s;
            rb = b * c + a * s;
        }
        T ta = from_float<T>(ra), tb = from_float<T>(rb);
        h[j] = ta;
        h[j + half] = tb;
        if (head >= nq) {
            size_t dst = page_base + ((size_t)(head - nq) * page_size + in_page) * d;
            k_cache[dst + j] = ta;
            k_cache[dst + j + half] = tb;
        }
    }
    const T* vrow = row + (size_t)(nq + nkv) * d;
    for (int it = threadIdx.x; it < nkv * d; it += blockDim.x) {
        int head = it / d, i = it - head * d;
        v_cache[page_base + ((size_t)head * page_size + in_page) * d + i] = vrow[it];
    }
}

// The same by fours of values, two tokens a CTA with 128 threads each.  1,024 float32 tokens of 9 + 3 + 3 heads of 64 on a B200: 4.8 us
// a value a thread and launched after the end of the product before it, 3.8 here; the attention after it starts 1.1 us earlier too.
template <typename T>
__global__ void __launch_bounds__(256)
rope_store_quads_kernel(T* __restrict__ qkv, const int* __restrict__ token_pos, const int* __restrict__ token_seq,
                        const int* __restrict__ page_table, int table_cols, const float* __restrict__ cos_t,
                        const float* __restrict__ sin_t, T* __restrict__ k_cache, T* __restrict__ v_cache, int n_tokens, int nq,
                        int nkv, int d, int page_size, int rotate) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = threadIdx.x & 127, n = blockIdx.x * 2 + (threadIdx.x >> 7);
    const int pos = n < n_tokens ? token_pos[n] : -1;
    if (pos < 0) return;  // a padding row: nothing to rotate, nothing to store
    const int half = d >> 1, quads = half >> 2;
    T* row = qkv + (size_t)n * (nq + 2 * nkv) * d;
    size_t base = 0;
    if (nkv > 0) {
        const int page = page_table[(size_t)token_seq[n] * table_cols + pos / page_size];
        base = ((size_t)page * nkv * page_size + pos % page_size) * d;
    }
    const int turned = (nq + nkv) * quads;
    for (int it = t; it < turned + nkv * 2 * quads; it += 128) {
        if (it >= turned) {  // a value's quad
            const int head = (it - turned) / (2 * quads), i = (it - turned - head * 2 * quads) * 4;
            store4(v_cache + base + (size_t)head * page_size * d + i, load4(row + (size_t)(nq + nkv + head) * d + i));
            continue;
        }
        const int head = it / quads, j = (it - head * quads) * 4;
        T* h = row + (size_t)head * d + j;
        float4 a = load4(h), b = load4(h + half);
        if (rotate) {
            const float4 c = load4(cos_t + (size_t)pos * half + j), s = load4(sin_t + (size_t)pos * half + j);
            const float4 x = make_float4(a.x * c.x - b.x * s.x, a.y * c.y - b.y * s.y, a.z * c.z - b.z * s.z, a.w * c.w - b.w * s.w);
            b = make_float4(b.x * c.x + a.x * s.x, b.y * c.y + a.y * s.y, b.z * c.z + a.z * s.z, b.w * c.w + a.w * s.w);
            a = x;
        }
        store4(h, a);
        store4(h + half, b);
        if (head >= nq) {
            T* k = k_cache + base + (size_t)(head - nq) * page_size * d + j;
            store4(k, a);
            store4(k + half, b);
        }
    }
}


// ---------------------------------------------------------------------------
// RMS norm in groups: a row of `width` is cut into `groups` equal runs, each
// divided by its own sqrt(mean(run^2) + eps), and the whole multiplied by w.
// A warp per (row, group); a lane reads the same elements in both passes, so
// y may be x itself (float32 output).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
group_rmsnorm_kernel(const float* x, const int* __restrict__ rows,
                     const float* __restrict__ w, T* y, long long n_units, int width, int groups,
                     float eps) {
    pdl_wait();
    pdl_launch_dependents();
    long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= n_units) return;
    int lane = threadIdx.x & 31;
    long long r = unit / groups;
    int g = (int)(unit - r * groups), gw = width / groups;
    const float* in = x + (size_t)(rows ? rows[r] : r) * width + (size_t)g * gw;
    float ss = 0.f;
    for (int i = lane; i < gw; i += 32) ss = fmaf(in[i], in[i], ss);
    ss = warp_sum(ss);
    float s = 1.0f / sqrtf(ss / (float)gw + eps);
    T* out = y + (size_t)r * width + (size_t)g * gw;
    const float* wg = w + (size_t)g * gw;
    for (int i = lane; i < gw; i += 32) out[i] = from_float<T>((in[i] * s) * wg[i]);
}

// The same for groups of a multiple of four values, at most 128 Q: the run and its weights in registers.
template <typename T, int Q>
__global__ void __launch_bounds__(256)
group_rmsnorm_quads_kernel(const float* x, const int* __restrict__ rows, const float* __restrict__ w, T* y,
                           long long n_units, int width, int groups, float eps) {
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= n_units) {
        pdl_wait();
        pdl_launch_dependents();
        return;
    }
    const int lane = threadIdx.x & 31, gw = width / groups;
    const long long r = unit / groups;
    const int g = (int)(unit - r * groups);
    RowQuads<Q> weight, run;
    weight.load(w + (size_t)g * gw, gw >> 2, lane);  // (depend on no kernel)
    pdl_wait();
    pdl_launch_dependents();
    run.load(x + (size_t)(rows ? rows[r] : r) * width + (size_t)g * gw, gw >> 2, lane);
    const float s = 1.0f / sqrtf(warp_sum(run.squares()) / (float)gw + eps);
    T* out = y + (size_t)r * width + (size_t)g * gw;
#pragma unroll
    for (int j = 0; j < Q; ++j)
        if (lane + 32 * j < gw >> 2)
            store4(out + 4 * (lane + 32 * j),
                   make_float4((run.v[j].x * s) * weight.v[j].x, (run.v[j].y * s) * weight.v[j].y,
                               (run.v[j].z * s) * weight.v[j].z, (run.v[j].w * s) * weight.v[j].w));
}

template <typename T>
static cudaError_t launch_group_rmsnorm(const float* x, const int* rows, const float* w, T* y, long long units, int width,
                                        int groups, float eps, cudaStream_t stream) {
    const unsigned blocks = (unsigned)((units + 7) / 8);
    const int gw = width / groups;
    auto kernel = group_rmsnorm_kernel<T>;
    if (gw % 4 == 0 && gw <= 1024 && ((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) % 16 == 0)
        kernel = gw <= 128 ? group_rmsnorm_quads_kernel<T, 1> : gw <= 256 ? group_rmsnorm_quads_kernel<T, 2>
                 : gw <= 512 ? group_rmsnorm_quads_kernel<T, 4> : group_rmsnorm_quads_kernel<T, 8>;
    return launch_dependent(kernel, blocks, 256, 0, stream, x, rows, w, y, units, width, groups, eps);
}

// ---------------------------------------------------------------------------
// a += b, float32, elementwise: where two branches of a layer that ran side by side meet
// in the residual stream.
// ---------------------------------------------------------------------------
__global__ void add_rows_kernel(float* __restrict__ a, const float* __restrict__ b, size_t count4) {
    pdl_wait();
    pdl_launch_dependents();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count4) return;
    float4 x = reinterpret_cast<float4*>(a)[i], y = reinterpret_cast<const float4*>(b)[i];
    reinterpret_cast<float4*>(a)[i] = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
}

// ---------------------------------------------------------------------------
// out[n, i] = relu(u[n, i])^2 (* sigmoid(u[n, inter]) when `gated` > 0): the
// activation of an expert whose row of u carries, in column `inter`, the logit
// of a gate that scales the expert's whole output.  u float32 [n, inter + gated]
// (`gated` columns beyond the activation's: the gate, then padding).
// ---------------------------------------------------------------------------
// 2^log_lanes threads a row and four values a thread, as far apart, all asked for at once, the gate once a thread.  Rows
// of 1,024 values and more take a CTA of 256 threads each, shorter ones share it (a thread a value, its row by a division
// of 64 bits: 12.5 us for 2,048 rows of 1,408, 21 for 20,000 of 256, 17.7 for 65,536 of 64; now 5.0, 6.9 and 5.9; a CTA a
// row took 21 and 69 for the last two).
template <typename T, bool WIDE>
__global__ void __launch_bounds__(256)
relu2_gate_kernel(const float* __restrict__ u, T* __restrict__ out, long long n_rows, int inter, int gated, int log_lanes) {
    pdl_wait();
    pdl_launch_dependents();
    const int lanes = WIDE ? 256 : 1 << log_lanes;
    const size_t n = WIDE ? blockIdx.x : (size_t)blockIdx.x * (256 >> log_lanes) + (threadIdx.x >> log_lanes);
    if (!WIDE && n >= (size_t)n_rows) return;
    const float* row = u + n * (size_t)(inter + gated);
    const int i0 = blockIdx.y * lanes * 4 + (WIDE ? threadIdx.x : threadIdx.x & (lanes - 1));
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = i0 + e * lanes < inter ? row[i0 + e * lanes] : 0.f;
    const float scale = gated ? 1.0f / (1.0f + expf(-row[inter])) : 1.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float a = fmaxf(x[e], 0.f);
        float v = a * a;
        if (gated) v *= scale;
        if (i0 + e * lanes < inter) out[n * inter + i0 + e * lanes] = from_float<T>(v);
    }
}

// ---------------------------------------------------------------------------
// Rotation of a part of every head by frequencies given as a table: for each
// token n and head h, the `len` elements at src[n, h * src_head + src_off ...]
// go to dst[n, h * dst_head + dst_off ...]; the first `dims` of them are turned
// in pairs (i, i + dims / 2), or with `neighbours` (2i, 2i + 1), by the angle pos * freq[i]
// (float32), the rest pass.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void rope_part_kernel(const T* src, long long src_row, int src_head,  // (src may be dst itself)
                                 int src_off, T* dst, long long dst_row, int dst_head,
                                 int dst_off, const int* __restrict__ token_pos,
                                 const float* __restrict__ freq, int heads, int len, int dims,
                                 int neighbours) {
    pdl_wait();
    pdl_launch_dependents();
    int n = blockIdx.x;
    int pos = token_pos[n];
    int half = dims >> 1;
    int items = heads * (len - half);  // a pair, or one element beyond the turned ones
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        int h = it / (len - half), j = it - h * (len - half);
        const T* s = src + (size_t)n * src_row + (size_t)h * src_head + src_off;
        T* d = dst + (size_t)n * dst_row + (size_t)h * dst_head + dst_off;
        if (j < half) {
            const int i0 = neighbours ? 2 * j : j, i1 = neighbours ? 2 * j + 1 : j + half;
            float a = to_float(s[i0]), b = to_float(s[i1]);
            float ang = (float)(pos < 0 ? 0 : pos) * freq[j];
            float c = cosf(ang), sn = sinf(ang);
            d[i0] = from_float<T>(a * c - b * sn);
            d[i1] = from_float<T>(b * c + a * sn);
        } else {
            d[j + half] = s[j + half];
        }
    }
}

// The same where everything lies by fours: two tokens a CTA, 128 threads each, four pairs (two with `neighbours`) or four passing
// values a thread, a token's cosines and sines made once for all its heads.  3,359 tokens of 16 heads of 64 on a B200: 10.0 us a
// pair a thread, 4.4 here.
constexpr int kRopeTurns = 128;
template <typename T>
__global__ void __launch_bounds__(256)
rope_part_quads_kernel(const T* src, long long src_row, int src_head, int src_off, T* dst, long long dst_row, int dst_head,
                       int dst_off, const int* __restrict__ token_pos, const float* __restrict__ freq, int n_tokens, int heads,
                       int len, int dims, int neighbours) {
    __shared__ float2 turns[2][kRopeTurns];
    pdl_wait();
    pdl_launch_dependents();
    const int side = threadIdx.x >> 7, t = threadIdx.x & 127, n = blockIdx.x * 2 + side, half = dims >> 1;
    const int pos = n < n_tokens ? max(token_pos[n], 0) : 0;
    for (int i = t; i < half; i += 128) {
        const float ang = (float)pos * freq[i];
        turns[side][i] = make_float2(cosf(ang), sinf(ang));
    }
    __syncthreads();
    if (n >= n_tokens) return;
    // items of a head: turned quads (of both halves, or of neighbours), then passing ones
    const int turned = neighbours ? dims >> 2 : half >> 2, items = turned + ((len - dims) >> 2);
    for (int it = t; it < heads * items; it += 128) {
        const int h = it / items, j = it - h * items;
        const T* s = src + (size_t)n * src_row + (size_t)h * src_head + src_off;
        T* d = dst + (size_t)n * dst_row + (size_t)h * dst_head + dst_off;
        if (j >= turned) {
            const int at = dims + 4 * (j - turned);
            store4(d + at, load4(s + at));
        } else if (neighbours) {
            const float4 x = load4(s + 4 * j);
            const float2 f = turns[side][2 * j], g = turns[side][2 * j + 1];
            store4(d + 4 * j, make_float4(x.x * f.x - x.y * f.y, x.y * f.x + x.x * f.y, x.z * g.x - x.w * g.y, x.w * g.x + x.z * g.y));
        } else {
            const float4 a = load4(s + 4 * j), b = load4(s + half + 4 * j);
            const float2 f0 = turns[side][4 * j], f1 = turns[side][4 * j + 1], f2 = turns[side][4 * j + 2], f3 = turns[side][4 * j + 3];
            store4(d + 4 * j, make_float4(a.x * f0.x - b.x * f0.y, a.y * f1.x - b.y * f1.y, a.z * f2.x - b.z * f2.y, a.w * f3.x - b.w * f3.y));
            store4(d + half + 4 * j, make_float4(b.x * f0.x + a.x * f0.y, b.y * f1.x + a.y * f1.y, b.z * f2.x + a.z * f2.y, b.w * f3.x + a.w * f3.y));
        }
    }
}

}  // namespace nnis

using namespace nnis;

// A copy in either direction on the stream (pinned host memory on the host side),
// for the few bytes a decode step exchanges with the host: one call, no allocation.
NNIS_API int nnis_copy_async(void* dst, const void* src, long long bytes, cudaStream_t stream) {
    if (!dst || !src || bytes <= 0) return NNIS_ERR_ARGUMENT;
    cudaError_t e = cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDefault, stream);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_stream_synchronize(cudaStream_t stream) {
    cudaError_t e = cudaStreamSynchronize(stream);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_embed(const void* table, int dtype, const int* tokens, float* hidden,
                        int n_tokens, int width, int vocab, int* status, float scale, cudaStream_t stream) {
    if (n_tokens <= 0 || width <= 0 || vocab <= 0 || !status) return NNIS_ERR_ARGUMENT;
    int threads = width >= 256 ? 256 : 64;
    const bool quads = width % 4 == 0 && ((uintptr_t)table | (uintptr_t)hidden) % 16 == 0;
    if (quads && dtype == NNIS_DTYPE_F32)
        embed_quads_kernel<float><<<n_tokens, 256, 0, stream>>>((const float*)table, tokens, hidden, width / 4, vocab,
                                                                status, scale);
    else if (quads && dtype == NNIS_DTYPE_BF16)
        embed_quads_kernel<bf16><<<n_tokens, 256, 0, stream>>>((const bf16*)table, tokens, hidden, width / 4, vocab,
                                                               status, scale);
    else if (dtype == NNIS_DTYPE_F32)
        embed_kernel<float><<<n_tokens, threads, 0, stream>>>((const float*)table, tokens, hidden,
                                                              n_tokens, width, vocab, status, scale);
    else if (dtype == NNIS_DTYPE_BF16)
        embed_kernel<bf16><<<n_tokens, threads, 0, stream>>>((const bf16*)table, tokens, hidden,
                                                             n_tokens, width, vocab, status, scale);
    else
        return NNIS_ERR_UNSUPPORTED;
    NNIS_RETURN_LAUNCH();
}

template <typename T>
static auto rmsnorm_of(int width) {
    return width <= 1024 ? rmsnorm_quads_kernel<T, 1> : width <= 2048 ? rmsnorm_quads_kernel<T, 2>
           : width <= 4096 ? rmsnorm_quads_kernel<T, 4> : rmsnorm_quads_kernel<T, 8>;
}

// `pdl`: launch as a programmatic dependent of the kernel before it on the stream
// (the kernel waits for that kernel's results itself).
NNIS_API int nnis_rmsnorm(const float* x, const int* rows, const float* w, void* y, int out_dtype,
                          int n_rows, int width, float eps, int pdl, cudaStream_t stream) {
    if (n_rows <= 0 || width <= 0 || !(eps > 0.f)) return NNIS_ERR_ARGUMENT;
    // many rows of moderate width on 16-byte boundaries: a warp per row
    const bool quads = width % 4 == 0 && width <= 8192 && ((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) % 16 == 0;
    const bool by_rows = n_rows >= 64 && quads && width <= 1024;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(by_rows ? (n_rows + 7) / 8 : n_rows);
    cfg.blockDim = dim3(quads ? 256 : (width >= 1024 ? 256 : (width >= 256 ? 128 : 32)));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaError_t e;
    if (out_dtype == NNIS_DTYPE_F32)
        e = by_rows ? cudaLaunchKernelEx(&cfg, rmsnorm_rows_kernel<float>, x, rows, w, (float*)y, n_rows, width, eps, trace_slot("rmsnorm rows"))
                    : cudaLaunchKernelEx(&cfg, quads ? rmsnorm_of<float>(width) : rmsnorm_kernel<float>, x, rows, w, (float*)y, width, eps);
    else if (out_dtype == NNIS_DTYPE_BF16)
        e = by_rows ? cudaLaunchKernelEx(&cfg, rmsnorm_rows_kernel<bf16>, x, rows, w, (bf16*)y, n_rows, width, eps, trace_slot("rmsnorm rows"))
                    : cudaLaunchKernelEx(&cfg, quads ? rmsnorm_of<bf16>(width) : rmsnorm_kernel<bf16>, x, rows, w, (bf16*)y, width, eps);
    else
        return NNIS_ERR_UNSUPPORTED;
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_silu_mul(const float* gate_up, void* out, int out_dtype, long long n_rows,
                           int inter, cudaStream_t stream) {
    if (n_rows <= 0 || inter <= 0) return NNIS_ERR_ARGUMENT;
    size_t total = (size_t)n_rows * inter;
    unsigned blocks = (unsigned)((total + 255) / 256);
    if (out_dtype == NNIS_DTYPE_F32)
        gate_mul_kernel<float, false><<<blocks, 256, 0, stream>>>(gate_up, (float*)out, n_rows, inter);
    else if (out_dtype == NNIS_DTYPE_BF16)
        gate_mul_kernel<bf16, false><<<blocks, 256, 0, stream>>>(gate_up, (bf16*)out, n_rows, inter);
    else
        return NNIS_ERR_UNSUPPORTED;
    NNIS_RETURN_LAUNCH();
}

NNIS_API int nnis_gelu_mul(const float* gate_up, void* out, int out_dtype, long long n_rows, int inter,
                           cudaStream_t stream) {
    if (n_rows <= 0 || inter <= 0) return NNIS_ERR_ARGUMENT;
    size_t total = (size_t)n_rows * inter;
    unsigned blocks = (unsigned)((total + 255) / 256);
    if (out_dtype == NNIS_DTYPE_F32)
        gate_mul_kernel<float, true><<<blocks, 256, 0, stream>>>(gate_up, (float*)out, n_rows, inter);
    else if (out_dtype == NNIS_DTYPE_BF16)
        gate_mul_kernel<bf16, true><<<blocks, 256, 0, stream>>>(gate_up, (bf16*)out, n_rows, inter);
    else
        return NNIS_ERR_UNSUPPORTED;
    NNIS_RETURN_LAUNCH();
}

NNIS_API int nnis_rope_store(void* qkv, int dtype, const int* token_pos, const int* token_seq,
                             const int* page_table, int table_cols, const float* cos_t,
                             const float* sin_t, void* k_cache, void* v_cache, int n_tokens, int nq,
                             int nkv, int d, int page_size, int rotate, cudaStream_t stream) {
    if (n_tokens <= 0 || nq < 0 || nkv < 0 || nq + nkv == 0 || d <= 0 || (d & 1))
        return NNIS_ERR_ARGUMENT;
    if (nkv > 0 && (!page_table || !k_cache || !v_cache || page_size <= 0 || table_cols <= 0))
        return NNIS_ERR_ARGUMENT;
    if (rotate && (!cos_t || !sin_t)) return NNIS_ERR_ARGUMENT;
    const uintptr_t rows = (uintptr_t)qkv | (uintptr_t)k_cache | (uintptr_t)v_cache;
    const uintptr_t turns = rotate ? (uintptr_t)cos_t | (uintptr_t)sin_t : 0;
    // A token of fewer than 64 items leaves most of its 128 threads idle, which many tokens feel: us in general / by fours,
    // 2 + 1 + 1 heads of 64 (40 items), bfloat16, 740 tokens 2.71 / 2.50, 1,024 2.84 / 3.01, 3,001 3.95 / 4.56; 2 + 2 + 2
    // heads (64 items) 3,001 5.12 / 4.06.
    const bool pays = (nq + nkv) * (d / 8) + nkv * (d / 4) >= 64 || n_tokens <= 5LL * device_sms();
    if (pays && d % 8 == 0 && turns % 16 == 0 && rows % (dtype == NNIS_DTYPE_F32 ? 16 : 8) == 0 &&
        (dtype == NNIS_DTYPE_F32 || dtype == NNIS_DTYPE_BF16)) {
        const unsigned blocks = (unsigned)(((long long)n_tokens + 1) / 2);
        const cudaError_t e = dtype == NNIS_DTYPE_F32
            ? launch_dependent(rope_store_quads_kernel<float>, blocks, 256, 0, stream, (float*)qkv, token_pos, token_seq, page_table, table_cols,
                               cos_t, sin_t, (float*)k_cache, (float*)v_cache, n_tokens, nq, nkv, d, page_size, rotate)
            : launch_dependent(rope_store_quads_kernel<bf16>, blocks, 256, 0, stream, (bf16*)qkv, token_pos, token_seq, page_table, table_cols,
                               cos_t, sin_t, (bf16*)k_cache, (bf16*)v_cache, n_tokens, nq, nkv, d, page_size, rotate);
        return e == cudaSuccess ? NNIS_OK : (int)e;
    }
    int work = (nq + nkv) * (d / 2);
    int threads = work >= 256 ? 256 : (work >= 128 ? 128 : 64);
    if (dtype == NNIS_DTYPE_F32)
        rope_store_kernel<float><<<n_tokens, threads, 0, stream>>>(
            (float*)qkv, token_pos, token_seq, page_table, table_cols, cos_t, sin_t,
            (float*)k_cache, (float*)v_cache, nq, nkv, d, page_size, rotate);
    else if (dtype == NNIS_DTYPE_BF16)
        rope_store_kernel<bf16><<<n_tokens, threads, 0, stream>>>(
            (bf16*)qkv, token_pos, token_seq, page_table, table_cols, cos_t, sin_t, (bf16*)k_cache,
            (bf16*)v_cache, nq, nkv, d, page_size, rotate);
    else
        return NNIS_ERR_UNSUPPORTED;
    NNIS_RETURN_LAUNCH();
}

NNIS_API int nnis_group_rmsnorm(const float* x, const int* rows, const float* w, void* y,
                                int out_dtype, int n_rows, int width, int groups, float eps,
                                cudaStream_t stream) {
    if (n_rows <= 0 || width <= 0 || groups <= 0 || width % groups || !(eps > 0.f))
        return NNIS_ERR_ARGUMENT;
    long long units = (long long)n_rows * groups;
    cudaError_t e;
    if (out_dtype == NNIS_DTYPE_F32)
        e = launch_group_rmsnorm(x, rows, w, (float*)y, units, width, groups, eps, stream);
    else if (out_dtype == NNIS_DTYPE_BF16)
        e = launch_group_rmsnorm(x, rows, w, (bf16*)y, units, width, groups, eps, stream);
    else
        return NNIS_ERR_UNSUPPORTED;
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_relu2_gate(const float* u, void* out, int out_dtype, long long n_rows, int inter,
                             int gated, cudaStream_t stream) {
    if (n_rows <= 0 || inter <= 0 || gated < 0) return NNIS_ERR_ARGUMENT;
    int log_lanes = 3;
    while (log_lanes < 8 && (4 << log_lanes) < inter) ++log_lanes;
    const long long rows = 256 >> log_lanes, blocks = (n_rows + rows - 1) / rows;
    const dim3 grid((unsigned)blocks, (unsigned)(((long long)inter + (4 << log_lanes) - 1) / (4 << log_lanes)));
    if (blocks > 0x7fffffffLL || grid.y > 65535) return NNIS_ERR_UNSUPPORTED;
    cudaError_t e;
    if (out_dtype == NNIS_DTYPE_F32)
        e = launch_dependent(log_lanes == 8 ? relu2_gate_kernel<float, true> : relu2_gate_kernel<float, false>, grid, 256, 0,
                             stream, u, (float*)out, n_rows, inter, gated, log_lanes);
    else if (out_dtype == NNIS_DTYPE_BF16)
        e = launch_dependent(log_lanes == 8 ? relu2_gate_kernel<bf16, true> : relu2_gate_kernel<bf16, false>, grid, 256, 0,
                             stream, u, (bf16*)out, n_rows, inter, gated, log_lanes);
    else
        return NNIS_ERR_UNSUPPORTED;
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_rope_part(const void* src, long long src_row, int src_head, int src_off, void* dst,
                            long long dst_row, int dst_head, int dst_off, const int* token_pos,
                            const float* freq, int n_tokens, int heads, int len, int dims, int neighbours,
                            int dtype, cudaStream_t stream) {
    if (n_tokens <= 0 || heads <= 0 || len <= 0 || dims < 0 || (dims & 1) || dims > len || !freq)
        return NNIS_ERR_ARGUMENT;
    // (every head's part starts by fours, and so do its halves and what passes)
    // (short steps are over before the barrier behind the angles pays.  us in general / by fours, bfloat16, halves: 16
    // heads of 64, 8 tokens 1.75 / 1.67 (float32 1.69 / 1.69), 256 2.10 / 1.85; 8 heads 128 tokens 1.54 / 1.79, 512 1.89 /
    // 1.93, 740 2.55 / 1.96; neighbours: 16 heads 8 tokens 1.74 / 1.99, 296 2.10 / 2.16, 512 2.66 / 2.30; 12 heads 444
    // tokens 2.14 / 2.29, 512 2.39 / 2.26; a head of 64, halves: 1,536 tokens 1.91 / 1.93, 2,560 2.98 / 2.92)
    const bool pays = (long long)n_tokens * heads * len >= (neighbours ? 3LL << 17 : 1LL << 18) || n_tokens > 16LL * device_sms();
    const bool quads = pays && len % 4 == 0 && dims % (neighbours ? 4 : 8) == 0 && dims / 2 <= kRopeTurns &&
                       !((src_row | dst_row | src_head | dst_head | src_off | dst_off) & 3) &&
                       ((uintptr_t)src | (uintptr_t)dst) % (dtype == NNIS_DTYPE_F32 ? 16 : 8) == 0;
    if (quads && (dtype == NNIS_DTYPE_F32 || dtype == NNIS_DTYPE_BF16)) {
        const unsigned blocks = (unsigned)((n_tokens + 1) / 2);
        const cudaError_t q = dtype == NNIS_DTYPE_F32
            ? launch_dependent(rope_part_quads_kernel<float>, blocks, 256, 0, stream, (const float*)src, src_row, src_head, src_off,
                               (float*)dst, dst_row, dst_head, dst_off, token_pos, freq, n_tokens, heads, len, dims, neighbours)
            : launch_dependent(rope_part_quads_kernel<bf16>, blocks, 256, 0, stream, (const bf16*)src, src_row, src_head, src_off,
                               (bf16*)dst, dst_row, dst_head, dst_off, token_pos, freq, n_tokens, heads, len, dims, neighbours);
        return q == cudaSuccess ? NNIS_OK : (int)q;
    }
    int work = heads * (len - dims / 2);
    int threads = work >= 256 ? 256 : (work >= 128 ? 128 : 64);
    cudaError_t e;
    if (dtype == NNIS_DTYPE_F32)
        e = launch_dependent(rope_part_kernel<float>, n_tokens, threads, 0, stream, (const float*)src, src_row,
                             src_head, src_off, (float*)dst, dst_row, dst_head, dst_off, token_pos, freq, heads,
                             len, dims, neighbours);
    else if (dtype == NNIS_DTYPE_BF16)
        e = launch_dependent(rope_part_kernel<bf16>, n_tokens, threads, 0, stream, (const bf16*)src, src_row,
                             src_head, src_off, (bf16*)dst, dst_row, dst_head, dst_off, token_pos, freq, heads,
                             len, dims, neighbours);
    else
        return NNIS_ERR_UNSUPPORTED;
    return e == cudaSuccess ? NNIS_OK : (int)e;
}

NNIS_API int nnis_add_rows(float* a, const float* b, long long count, cudaStream_t stream) {
    if (!a || !b || count <= 0 || count % 4 || ((uintptr_t)a | (uintptr_t)b) % 16) return NNIS_ERR_ARGUMENT;
    size_t count4 = (size_t)count / 4;
    cudaError_t e = launch_dependent(add_rows_kernel, (unsigned)((count4 + 255) / 256), 256, 0, stream, a, b, count4);
    return e == cudaSuccess ? NNIS_OK : (int)e;
}
