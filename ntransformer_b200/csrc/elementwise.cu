// elementwise.cu — activation quantiser, RMSNorm, RoPE, KV-cache write, SwiGLU, residual adds, softmax,
// embedding gather.  Reference kernels K10-K15, K19-K21 (src/cuda/{rmsnorm,rotary,elementwise,softmax}.cu,
// gemm.cu:699-725, attention.cu:316-342).
//
// This file is compiled with --use_fast_math like the reference (CMakeLists.txt:20) and writes the
// transcendental expressions in the same form (1.0f / powf, cosf/sinf, g / (1 + expf(-g)), rsqrtf) so they
// lower to the same approximate instructions: greedy-token parity depends on it.
// Anything that must stay IEEE uses explicit *_rn intrinsics.
#include "kernels_internal.h"
#include "xquant.cuh"
#include "ring.cuh"
#include <cuda_fp16.h>
#include <cfloat>
#include <atomic>

namespace nt { namespace b200 {

static std::atomic<unsigned long long> g_launches{0};
unsigned long long launch_count() { return g_launches.load(); }
void count_launch(int n) { g_launches.fetch_add((unsigned long long)n); }
static std::atomic<unsigned long long> g_programmatic{0};
unsigned long long programmatic_count() { return g_programmatic.load(); }
void count_programmatic() { g_programmatic.fetch_add(1); }
static thread_local Launches t_launches = Launches::Boundary;
Launches launches() { return t_launches; }
LaunchScope::LaunchScope(Launches m) : was(t_launches) { t_launches = m; }
LaunchScope::~LaunchScope() { t_launches = was; }

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
// Block-wide sum / max over blockDim.x (multiple of 32, <= 1024) threads; result valid in every thread.
__device__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    float t = (lane < nw) ? red[lane] : 0.f;
    return warp_sum(t);
}
__device__ float block_max(float v, float* red) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    float t = (lane < nw) ? red[lane] : -FLT_MAX;
    return warp_max(t);
}

__global__ void quantize_x_kernel(const float* __restrict__ x, int8_t* __restrict__ xq, int K) {
    pdl_launch_dependents();
    pdl_wait();
    x = behind_wait(x);
    const int blk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (blk * 32 >= K) return;
    quantize_block32(x[blk * 32 + lane], blk, lane, xq, K);
}

// ---- RMSNorm: y = x * rsqrtf(mean(x^2) + eps) * w, one CTA per row (rmsnorm.cu:17-70) ----
// One row is all latency.  Up to KEEP elements to a thread, x and w are fetched once and together and stay in registers; longer rows read both again behind the sum.
template <bool HALF_OUT, int KEEP>
__global__ void __launch_bounds__(1024) rmsnorm_kernel(void* __restrict__ yv, const float* __restrict__ xin,
                                                       const float* __restrict__ w, int hidden, float eps) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[32];
    const float* x = behind_wait(xin) + (size_t)blockIdx.x * hidden;
    w = behind_wait(w);
    auto store = [&](int i, float v) {
        if (HALF_OUT) reinterpret_cast<__half*>(yv)[(size_t)blockIdx.x * hidden + i] = __float2half(v);
        else reinterpret_cast<float*>(yv)[(size_t)blockIdx.x * hidden + i] = v;
    };
    float ss = 0.f;
    if constexpr (KEEP > 0) {
        float xs[KEEP], ws[KEEP];
#pragma unroll
        for (int j = 0; j < KEEP; j++) { const int i = threadIdx.x + j * blockDim.x; xs[j] = i < hidden ? x[i] : 0.f; }
#pragma unroll
        for (int j = 0; j < KEEP; j++) { const int i = threadIdx.x + j * blockDim.x; ws[j] = i < hidden ? w[i] : 0.f; }
#pragma unroll
        for (int j = 0; j < KEEP; j++) ss += xs[j] * xs[j];
        const float rms_inv = rsqrtf(block_sum(ss, red) / hidden + eps);
#pragma unroll
        for (int j = 0; j < KEEP; j++) { const int i = threadIdx.x + j * blockDim.x; if (i < hidden) store(i, xs[j] * rms_inv * ws[j]); }
    } else {
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) { float v = x[i]; ss += v * v; }
        const float rms_inv = rsqrtf(block_sum(ss, red) / hidden + eps);
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) store(i, x[i] * rms_inv * w[i]);
    }
}
inline int norm_threads(int hidden) { return hidden <= 1024 ? 256 : hidden <= 4096 ? 512 : 1024; }
template <bool HALF_OUT>
void launch_rmsnorm_rows(void* y, const float* x, const float* w, int rows, int hidden, float eps, cudaStream_t s) {
    constexpr int KEEP = 8;                                        // rows to 8192, the widest model's
    const int threads = norm_threads(hidden);
    launch_k_pdl(true, hidden <= KEEP * threads ? rmsnorm_kernel<HALF_OUT, KEEP> : rmsnorm_kernel<HALF_OUT, 0>, dim3(rows), dim3(threads), 0, s, y, x, w, hidden, eps);
    count_launch();
}

// Multi-CTA RMSNorm + activation quantiser for the decode step: every CTA recomputes the (cheap, L2-resident)
// sum of squares in the same order, so all CTAs derive the bit-identical rms_inv, then quantises 8 of the
// row's 32-element blocks.  ~3 us instead of the 13.7 us of the single-CTA form on hidden = 8192.
__global__ void __launch_bounds__(256) rmsnorm_xq_kernel(float* __restrict__ y, int8_t* __restrict__ xq, const float* __restrict__ x,
                                                         const float* __restrict__ w, int hidden, float eps) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    float ss = 0.f;
    for (int i = threadIdx.x; i < hidden; i += 256) { float v = x[i]; ss += v * v; }
    ss = block_sum(ss, red);
    const float rms_inv = rsqrtf(ss / hidden + eps);
    const int blk = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (blk * 32 >= hidden) return;
    const int e = blk * 32 + lane;
    const float v = x[e] * rms_inv * w[e];
    if (y) y[e] = v;
    quantize_block32(v, blk, lane, xq, hidden);
}

// ---- RoPE (rotary.cu:16-107) ----
template <bool INTERLEAVED>
__global__ void rope_kernel(float* __restrict__ q, float* __restrict__ k, const int* __restrict__ positions, int seq_len,
                            int n_heads, int n_kv_heads, int head_dim, float theta_base, float freq_scale) {
    pdl_launch_dependents();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int half_dim = head_dim / 2;
    const int total_q = seq_len * n_heads * half_dim, total_k = seq_len * n_kv_heads * half_dim;
    if (idx >= total_q + total_k) return;
    const bool is_key = idx >= total_q;
    const int li = is_key ? idx - total_q : idx;
    const int n_h = is_key ? n_kv_heads : n_heads;
    const int pair = li % half_dim, head = (li / half_dim) % n_h, sp = li / (half_dim * n_h);
    const float freq = 1.0f / powf(theta_base, (2.0f * pair) / head_dim);
    pdl_wait();
    q = behind_wait(q); k = behind_wait(k);
    const int pos = behind_wait(positions)[sp];
    float angle = pos * freq * freq_scale;
    float c = cosf(angle), sn = sinf(angle);
    float* d = (is_key ? k : q) + (size_t)sp * n_h * head_dim + (size_t)head * head_dim;
    const int i0 = INTERLEAVED ? 2 * pair : pair, i1 = INTERLEAVED ? 2 * pair + 1 : pair + half_dim;
    float x0 = d[i0], x1 = d[i1];
    d[i0] = x0 * c - x1 * sn;
    d[i1] = x1 * c + x0 * sn;
}

// ---- KV-cache write: F32 -> F16 RN at [start_pos + s] (attention.cu:316-342) ----
// EACH elements to a thread, a block's width apart: a block costs its start and its wait, which long runs of one-element threads are bound by (copy of 64 M: 272 us, 184 without the
// wait)
template <int EACH>
__global__ void __launch_bounds__(256) kv_write_kernel(__half* __restrict__ kc, __half* __restrict__ vc, const float* __restrict__ k,
                                const float* __restrict__ v, int seq_len, int row /* n_kv * hd */, int start_pos, int max_seq) {
    pdl_launch_dependents();
    pdl_wait();
    k = behind_wait(k); v = behind_wait(v);
    const int i0 = blockIdx.x * (256 * EACH) + threadIdx.x;
    // rows behind the cache are silently dropped, like attention.cu:336
    const long long total = min((long long)seq_len * row, max(0ll, (long long)max_seq - start_pos) * row);
    float a[EACH], b[EACH];
#pragma unroll
    for (int e = 0; e < EACH; e++) { const int idx = i0 + 256 * e; if (idx < total) { a[e] = k[idx]; b[e] = v[idx]; } }
#pragma unroll
    for (int e = 0; e < EACH; e++) {
        const int idx = i0 + 256 * e;
        if (idx >= total) return;
        const int s = idx / row, c = idx - s * row;
        kc[(size_t)(start_pos + s) * row + c] = __float2half(a[e]);
        vc[(size_t)(start_pos + s) * row + c] = __float2half(b[e]);
    }
}

// Both for a run of tokens from start_pos on, one block to a token: q in place, k and v to the cache (k itself stays as it was).  A thread keeps four pairs of a head
// and their angles for every head it meets, where rope_kernel formed them anew for each (bound by powf, cosf and sinf): 8B heads, 2048 tokens 15.3 us, 29.5 + 10 for the two.
__global__ void __launch_bounds__(256) rope_kv_rows_kernel(float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, __half* __restrict__ kc,
                                                           __half* __restrict__ vc, int start_pos, int n_heads, int n_kv, int head_dim, float theta_base, float freq_scale,
                                                           int max_seq) {
    pdl_launch_dependents();
    pdl_wait();
    q = behind_wait(q); k = behind_wait(k); v = behind_wait(v);
    const int half_dim = head_dim / 2, per_head = half_dim / 4, pos = start_pos + blockIdx.x;
    const int pair = threadIdx.x % per_head * 4;                   // 256 is a multiple of per_head
    float c[4], sn[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float freq = 1.0f / powf(theta_base, (2.0f * (pair + i)) / head_dim);
        const float angle = pos * freq * freq_scale;
        c[i] = cosf(angle); sn[i] = sinf(angle);
    }
    const size_t row = (size_t)pos * n_kv * head_dim;
    auto halves = [](float a, float b, float d, float e) {
        const __half2 x = __floats2half2_rn(a, b), y = __floats2half2_rn(d, e);
        return make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
    };
    for (int h = threadIdx.x / per_head; h < n_heads + n_kv; h += 256 / per_head) {
        const bool is_key = h >= n_heads;
        if (is_key && pos >= max_seq) break;
        const float* src = is_key ? k + ((size_t)blockIdx.x * n_kv + h - n_heads) * head_dim : q + ((size_t)blockIdx.x * n_heads + h) * head_dim;
        const float4 a = *reinterpret_cast<const float4*>(src + pair), b = *reinterpret_cast<const float4*>(src + pair + half_dim);
        const float x0[4] = {a.x, a.y, a.z, a.w}, x1[4] = {b.x, b.y, b.z, b.w};
        float r0[4], r1[4];
#pragma unroll
        for (int i = 0; i < 4; i++) { r0[i] = x0[i] * c[i] - x1[i] * sn[i]; r1[i] = x1[i] * c[i] + x0[i] * sn[i]; }
        if (is_key) {
            __half* d = kc + row + (size_t)(h - n_heads) * head_dim + pair;
            *reinterpret_cast<uint2*>(d) = halves(r0[0], r0[1], r0[2], r0[3]);
            *reinterpret_cast<uint2*>(d + half_dim) = halves(r1[0], r1[1], r1[2], r1[3]);
        } else {
            float* d = q + ((size_t)blockIdx.x * n_heads + h) * head_dim + pair;
            *reinterpret_cast<float4*>(d) = make_float4(r0[0], r0[1], r0[2], r0[3]);
            *reinterpret_cast<float4*>(d + half_dim) = make_float4(r1[0], r1[1], r1[2], r1[3]);
        }
    }
    if (pos < max_seq)
        for (int i = threadIdx.x * 4; i < n_kv * head_dim; i += 1024) {
            const float4 a = *reinterpret_cast<const float4*>(v + (size_t)blockIdx.x * n_kv * head_dim + i);
            *reinterpret_cast<uint2*>(vc + row + i) = halves(a.x, a.y, a.z, a.w);
        }
}

// Decode-step fusion of K14 + K15: rotate q and k (pairs (i, i + hd/2)), then store F16 k, v at cache row *pos_dev.
__global__ void rope_kv_decode_kernel(float* __restrict__ q, float* __restrict__ k, const float* __restrict__ v,
                                      __half* __restrict__ kc, __half* __restrict__ vc, const int* __restrict__ pos_dev,
                                      int n_heads, int n_kv, int head_dim, float theta_base, float freq_scale, int max_seq) {
    pdl_launch_dependents();
    pdl_wait();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int half_dim = head_dim / 2;
    const int total_q = n_heads * half_dim, total_k = n_kv * half_dim;
    if (idx >= total_q + total_k) return;
    const bool is_key = idx >= total_q;
    const int li = is_key ? idx - total_q : idx;
    const int pair = li % half_dim, head = li / half_dim;
    const int pos = *pos_dev;
    float freq = 1.0f / powf(theta_base, (2.0f * pair) / head_dim);
    float angle = pos * freq * freq_scale;
    float c = cosf(angle), sn = sinf(angle);
    float* d = (is_key ? k : q) + (size_t)head * head_dim;
    float x0 = d[pair], x1 = d[pair + half_dim];
    float r0 = x0 * c - x1 * sn, r1 = x1 * c + x0 * sn;
    d[pair] = r0;
    d[pair + half_dim] = r1;
    if (is_key && pos < max_seq) {
        const size_t row = (size_t)pos * n_kv * head_dim + (size_t)head * head_dim;
        kc[row + pair] = __float2half(r0);
        kc[row + pair + half_dim] = __float2half(r1);
        vc[row + pair] = __float2half(v[(size_t)head * head_dim + pair]);
        vc[row + pair + half_dim] = __float2half(v[(size_t)head * head_dim + pair + half_dim]);
    }
}

__global__ void silu_mul_kernel(float* __restrict__ out, const float* __restrict__ gate, const float* __restrict__ up, int n) {
    pdl_launch_dependents();
    pdl_wait();
    gate = behind_wait(gate); up = behind_wait(up);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { float g = gate[i]; float silu = g / (1.0f + expf(-g)); out[i] = silu * up[i]; }
}
__global__ void add_kernel(float* out, const float* a, const float* b, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = a[i] + b[i];
}
template <int EACH>
__global__ void __launch_bounds__(256) copy_kernel(float* __restrict__ dst, const float* __restrict__ src, int n) {
    pdl_launch_dependents();
    pdl_wait();
    src = behind_wait(src);
    const int i0 = blockIdx.x * (256 * EACH) + threadIdx.x;
    float a[EACH];
#pragma unroll
    for (int e = 0; e < EACH; e++) if (i0 + 256 * e < n) a[e] = src[i0 + 256 * e];
#pragma unroll
    for (int e = 0; e < EACH; e++) if (i0 + 256 * e < n) dst[i0 + 256 * e] = a[e];
}
// single-block cosine similarity (elementwise.cu:46-84): dot / (|a||b|), 0 when the denominator is <= 1e-8
__global__ void __launch_bounds__(1024) cosine_kernel(float* result, const float* __restrict__ a, const float* __restrict__ b, int n) {
    __shared__ float red[32];
    float dot = 0.f, na = 0.f, nb = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) { float x = a[i], y = b[i]; dot += x * y; na += x * x; nb += y * y; }
    dot = block_sum(dot, red); na = block_sum(na, red); nb = block_sum(nb, red);
    if (threadIdx.x == 0) { float denom = sqrtf(na) * sqrtf(nb); *result = (denom > 1e-8f) ? dot / denom : 0.0f; }
}

// ---- row softmax, optional bool mask (softmax.cu:17-162): masked-out entries -> 0 ----
template <bool MASKED>
__global__ void __launch_bounds__(1024) softmax_kernel(float* __restrict__ out, const float* __restrict__ in,
                                                       const bool* __restrict__ mask, int cols) {
    __shared__ float red[32];
    const float* x = in + (size_t)blockIdx.x * cols;
    const bool* mk = (MASKED && mask) ? mask + (size_t)blockIdx.x * cols : nullptr;
    float* y = out + (size_t)blockIdx.x * cols;
    float mx = -FLT_MAX;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) if (!mk || mk[i]) mx = fmaxf(mx, x[i]);
    mx = block_max(mx, red);
    float sum = 0.f;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
        float e = (!mk || mk[i]) ? expf(x[i] - mx) : 0.f;
        y[i] = e;
        sum += e;
    }
    sum = block_sum(sum, red);
    float inv = (sum > 0.f) ? 1.0f / sum : 0.f;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) y[i] *= inv;
}

// ---- C[M,N] = A[M,K] . B[N,K]^T in F32 (gemm.cu:677-694; dead code in the reference) ----
__global__ void gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ B, int M, int N, int K) {
    __shared__ float sa[16][17], sb[16][17];
    const int row = blockIdx.y * 16 + threadIdx.y, col = blockIdx.x * 16 + threadIdx.x;
    float acc = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        int ka = k0 + threadIdx.x;
        sa[threadIdx.y][threadIdx.x] = (row < M && ka < K) ? A[(size_t)row * K + ka] : 0.f;
        int brow = blockIdx.x * 16 + threadIdx.y;
        sb[threadIdx.y][threadIdx.x] = (brow < N && ka < K) ? B[(size_t)brow * K + ka] : 0.f;
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; kk++) acc = fmaf(sa[threadIdx.y][kk], sb[threadIdx.x][kk], acc);
        __syncthreads();
    }
    if (row < M && col < N) C[(size_t)row * N + col] = acc;
}

// ---- embedding gather + dequant on the GPU: one CTA per token ----
__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ float dequant_at(const uint8_t* row, int dt, int i) {
    switch (dt) {
        case (int)DType::F32: return reinterpret_cast<const float*>(row)[i];
        case (int)DType::F16: return h2f(reinterpret_cast<const uint16_t*>(row)[i]);
        case (int)DType::BF16: return __uint_as_float((unsigned)reinterpret_cast<const uint16_t*>(row)[i] << 16);
        case (int)DType::Q8_0: {
            const uint8_t* b = row + (size_t)(i >> 5) * 34;
            return h2f(*reinterpret_cast<const uint16_t*>(b)) * (float)(int8_t)b[2 + (i & 31)];
        }
        case (int)DType::Q4_0: {
            const uint8_t* b = row + (size_t)(i >> 5) * 18;
            int j = i & 31;
            uint8_t byte = b[2 + (j & 15)];
            int qv = (j < 16) ? (byte & 15) : (byte >> 4);
            return h2f(*reinterpret_cast<const uint16_t*>(b)) * (float)(qv - 8);
        }
        case (int)DType::Q4_K_M: {
            const uint8_t* b = row + (size_t)(i >> 8) * 144;
            int n = i & 255, chunk = n >> 6, l = n & 31, hi = (n >> 5) & 1;
            int is = 2 * chunk + hi;
            const uint8_t* s = b + 4;
            int sc, m;
            if (is < 4) { sc = s[is] & 63; m = s[is + 4] & 63; }
            else { sc = (s[is + 4] & 15) | ((s[is - 4] >> 6) << 4); m = (s[is + 4] >> 4) | ((s[is] >> 6) << 4); }
            uint8_t byte = b[16 + chunk * 32 + l];
            int qv = hi ? (byte >> 4) : (byte & 15);
            float d = h2f(*reinterpret_cast<const uint16_t*>(b)), dmin = h2f(*reinterpret_cast<const uint16_t*>(b + 2));
            return (d * sc) * qv - dmin * m;
        }
        case (int)DType::Q6_K: {
            const uint8_t* b = row + (size_t)(i >> 8) * 210;
            int n = i & 255, hf = n >> 7, r = n & 127, run = r >> 5, l = r & 31;
            const uint8_t* ql = b + 64 * hf;
            const uint8_t* qh = b + 128 + 32 * hf;
            const int8_t* sc = reinterpret_cast<const int8_t*>(b + 192 + 8 * hf);
            uint8_t qb = ql[l + ((run & 1) ? 32 : 0)];
            int lo = (run >= 2) ? (qb >> 4) : (qb & 15);
            int q = (lo | (((qh[l] >> (2 * run)) & 3) << 4)) - 32;
            float d = h2f(*reinterpret_cast<const uint16_t*>(b + 208));
            return d * (float)sc[(l >> 4) + 2 * run] * q;
        }
        default: return 0.f;        // Q5_K table: zeros, as the reference (transformer.cpp:595-598)
    }
}
// A thread takes EACH elements, 256 apart, their fetches under way together (one block to a token walked its row 256 elements at a time, a trip to memory each: one
// token of 4096 in Q4_K 13 us, of 8192 23 us).
template <int EACH>
__global__ void __launch_bounds__(256) embed_kernel(float* __restrict__ out, const uint8_t* __restrict__ table, int dt, size_t row_bytes,
                                                    const int* __restrict__ tokens, int hidden) {
    pdl_launch_dependents();
    pdl_wait();
    const uint8_t* row = table + (size_t)tokens[blockIdx.x] * row_bytes;
    float v[EACH];
    const int i0 = blockIdx.y * 256 * EACH + threadIdx.x;
#pragma unroll
    for (int j = 0; j < EACH; j++) v[j] = i0 + 256 * j < hidden ? dequant_at(row, dt, i0 + 256 * j) : 0.f;
#pragma unroll
    for (int j = 0; j < EACH; j++) if (i0 + 256 * j < hidden) out[(size_t)blockIdx.x * hidden + i0 + 256 * j] = v[j];
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }
constexpr int WIDE_RUN = 1 << 18;      // elements from which a thread takes four: 148 SMs have a block of each kind then

}  // namespace

void quantize_x(const float* x, void* xq, int K, cudaStream_t s) {
    NT_CHECK(K % 128 == 0, "quantize_x: K must be a multiple of 128");
    launch_k_pdl(true, quantize_x_kernel, dim3(cdiv(K, 256)), dim3(256), 0, s, x, static_cast<int8_t*>(xq), K);
    count_launch();
}

void rmsnorm(float* y, const float* x, const float* w, int rows, int hidden, float eps, cudaStream_t s) {
    if (rows <= 0) return;
    launch_rmsnorm_rows<false>(y, x, w, rows, hidden, eps, s);
}
void rmsnorm_f16(void* y, const float* x, const float* w, int rows, int hidden, float eps, cudaStream_t s) {
    if (rows <= 0) return;
    launch_rmsnorm_rows<true>(y, x, w, rows, hidden, eps, s);
}
void rmsnorm_xq(float* y, void* xq, const float* x, const float* w, int hidden, float eps, cudaStream_t s) {
    NT_CHECK(hidden % 128 == 0, "rmsnorm_xq: hidden must be a multiple of 128");
    launch_k(rmsnorm_xq_kernel, dim3(cdiv(hidden / 32, 8)), dim3(256), 0, s, y, static_cast<int8_t*>(xq), x, w, hidden, eps);
    count_launch();
}
void rope(float* q, float* k, const int* positions, int seq_len, int n_heads, int n_kv_heads, int head_dim,
          float theta, float freq_scale, bool interleaved, cudaStream_t s) {
    int total = seq_len * (n_heads + n_kv_heads) * (head_dim / 2);
    if (total <= 0) return;
    launch_k_pdl(true, interleaved ? rope_kernel<true> : rope_kernel<false>, dim3(cdiv(total, 256)), dim3(256), 0, s, q, k, positions, seq_len, n_heads, n_kv_heads, head_dim,
                 theta, freq_scale);
    count_launch();
}
void copy_to_kv_cache(void* kc, void* vc, const float* k, const float* v, int seq_len, int n_kv, int hd,
                      int start_pos, int max_seq, cudaStream_t s) {
    int total = seq_len * n_kv * hd;
    if (total <= 0) return;
    const int each = total >= WIDE_RUN ? 4 : 1;
    launch_k_pdl(true, each == 4 ? kv_write_kernel<4> : kv_write_kernel<1>, dim3(cdiv(total, 256 * each)), dim3(256), 0, s, static_cast<__half*>(kc), static_cast<__half*>(vc), k, v, seq_len, n_kv * hd, start_pos, max_seq);
    count_launch();
}
bool rope_kv_rows(float* q, const float* k, const float* v, void* kc, void* vc, int tokens, int start_pos, int n_heads, int n_kv, int hd, float theta, float freq_scale,
                  int max_seq, cudaStream_t s) {
    if (hd != 64 && hd != 128 && hd != 256) return false;
    if (tokens <= 0) return true;
    launch_k_pdl(true, rope_kv_rows_kernel, dim3(tokens), dim3(256), 0, s, q, k, v, static_cast<__half*>(kc), static_cast<__half*>(vc), start_pos, n_heads, n_kv, hd, theta,
                 freq_scale, max_seq);
    count_launch();
    return true;
}
void rope_kv_decode(float* q, float* k, const float* v, void* kc, void* vc, const int* pos_dev, int n_heads, int n_kv,
                    int hd, float theta, float freq_scale, int max_seq, cudaStream_t s) {
    int total = (n_heads + n_kv) * (hd / 2);
    launch_k(rope_kv_decode_kernel, dim3(cdiv(total, 256)), dim3(256), 0, s, q, k, v, static_cast<__half*>(kc),
             static_cast<__half*>(vc), pos_dev, n_heads, n_kv, hd, theta, freq_scale, max_seq);
    count_launch();
}
void silu_mul(float* out, const float* gate, const float* up, int n, cudaStream_t s) {
    if (n <= 0) return;
    launch_k_pdl(true, silu_mul_kernel, dim3(cdiv(n, 256)), dim3(256), 0, s, out, gate, up, n);
    count_launch();
}
void add(float* out, const float* a, const float* b, int n, cudaStream_t s) {
    if (n <= 0) return;
    launch_k_pdl(true, add_kernel, dim3(cdiv(n, 256)), dim3(256), 0, s, out, a, b, n);
    count_launch();
}
void add_inplace(float* a, const float* b, int n, cudaStream_t s) { add(a, a, b, n, s); }
void add_bias(float* y, const float* b, int n, cudaStream_t s) { add(y, y, b, n, s); }
void copy(float* dst, const float* src, int n, cudaStream_t s) {
    if (n <= 0) return;
    const int each = n >= WIDE_RUN ? 4 : 1;
    launch_k_pdl(true, each == 4 ? copy_kernel<4> : copy_kernel<1>, dim3(cdiv(n, 256 * each)), dim3(256), 0, s, dst, src, n);
    count_launch();
}
void cosine_similarity(float* result, const float* a, const float* b, int n, cudaStream_t s) {
    cosine_kernel<<<1, 1024, 0, s>>>(result, a, b, n);
    count_launch();
}
void softmax(float* out, const float* in, int rows, int cols, cudaStream_t s) {
    if (rows <= 0) return;
    softmax_kernel<false><<<rows, norm_threads(cols), 0, s>>>(out, in, nullptr, cols);
    count_launch();
}
void masked_softmax(float* out, const float* in, const bool* mask, int rows, int cols, cudaStream_t s) {
    if (rows <= 0) return;
    softmax_kernel<true><<<rows, norm_threads(cols), 0, s>>>(out, in, mask, cols);
    count_launch();
}
void gemm_f32(float* C, const float* A, const float* B, int M, int N, int K, cudaStream_t s) {
    if (M <= 0 || N <= 0) return;
    dim3 block(16, 16), grid(cdiv(N, 16), cdiv(M, 16));
    gemm_f32_kernel<<<grid, block, 0, s>>>(C, A, B, M, N, K);
    count_launch();
}
void embed_rows(float* out, const void* table, DType dt, const int* tokens_dev, int n_tokens, int hidden, cudaStream_t s) {
    if (n_tokens <= 0) return;
    const int each = n_tokens < 16 ? 1 : 4;                        // a few tokens: more blocks than elements to a thread
    launch_k(each == 1 ? embed_kernel<1> : embed_kernel<4>, dim3(n_tokens, cdiv(hidden, 256 * each)), dim3(256), 0, s, out, static_cast<const uint8_t*>(table), (int)dt,
             dtype_row_size(dt, (size_t)hidden), tokens_dev, hidden);
    count_launch();
}

}}  // namespace nt::b200
