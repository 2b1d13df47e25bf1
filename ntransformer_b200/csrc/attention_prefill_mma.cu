// attention_prefill_mma.cu — causal GQA attention over a whole prompt chunk (prefill), sm_100a.
//
// Same contract as the reference's attention_prefill_kernel (src/cuda/attention.cu:216-311): F32 queries
// [seq][n_heads][hd], F16 KV cache [max_seq][n_kv][hd], query i attends keys 0..start_pos+i, softmax(q.k*scale).v.
// The reference (and csrc/attention.cu's prefill_kernel) re-reads the whole key range once per query; here a CTA owns
// 64 queries of one head and streams 64-key K/V tiles through shared memory (cp.async, double buffered), with the two
// contractions on the warp-level tensor-core path (mma.sync m16n8k16, F32 accumulate) and an online softmax in
// registers (flash-attention-2 data flow).  F32 operands are split into two F16 terms (q = hi + lo, p = hi + lo) so
// the result keeps ~22 mantissa bits and stays within the 2e-5 tolerance of the oracle.
//
// Prompts over an F16 cache take attention_prefill_tc.cu where that pays (attention.cu attention_prefill_tc_pays) and it takes them; this form is for the others.
// Calls over an F16 cache with fewer CTAs than SMs go in slices of their keys (attention.cu attention_prefill_slices_for), which a second launch joins.
// The same kernel serves windowed attention (csrc/attention_window.cu's rule: key j visible from position p iff j <= p and
// (p - j < window or j < keep)), optionally with soft-capped scores cap * tanh(s / cap) and a BF16 cache (BF: both MMAs take
// BF16 operands, the splits are BF16 pairs): a query block then walks only the key tiles of the kept prefix and of its window.
#include "kernels_internal.h"
#include "ring.cuh"
#include "attention_row.cuh"
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <algorithm>

namespace nt { namespace b200 {

namespace {

constexpr int BQ = 64, BKV = 64, PAD = 8;      // PAD halfs: row stride 272 B (hd 128) keeps LDS.32 / ldmatrix conflict-free

template <bool BF>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (BF)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// (x, y) -> packed F16 hi pair and lo pair with x = hi + lo to ~2^-22
template <bool BF>
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    if (BF) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        const float2 fb = __bfloat1622float2(b);
        const __nv_bfloat162 l = __floats2bfloat162_rn(x - fb.x, y - fb.y);
        hi = *reinterpret_cast<const uint32_t*>(&b);
        lo = *reinterpret_cast<const uint32_t*>(&l);
        return;
    }
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    hi = h2_bits(h);
    lo = h2_bits(__floats2half2_rn(x - f.x, y - f.y));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// HD: query / key head width, HDV: value head width.  maps > 1: blockIdx.y walks (head, map) pairs — map m of head h scores against
// map m of key head kvh (key rows [n_kv][maps][HD]) and sums kvh's one value row (value rows [n_kv][HDV]); n_heads counts the
// (head, map) pairs.  chunk > 0 replaces the window rule: key j visible from p iff j <= p and j / chunk == p / chunk.
// SLICED: blockIdx.z has a slice of the key tiles and leaves in parts its sums [slice][query][head][HDV], then (maximum, sum of weights) of each, for prefill_merge_kernel.
// Sums as in the form on tcgen05: each addition inside the tensor cores is cut off, so the high halves' products are summed over 64 channels and over a tile's 16 keys x 4
// at most before F32 takes them, the low halves' apart, and queries go in under a power of two per row.  Error against 64 bits over 40 tokens behind 965, 8 heads of 128:
// 3e-7; 7e-7 with scores and sums in one run each; 4e-7 on tcgen05.
__host__ __device__ constexpr int slice_tiles(int tiles, int slices) { return (tiles + slices - 1) / slices; }      // the last slices may have fewer, or none
template <int HD, int HDV, bool BF, bool SLICED>
__global__ void __launch_bounds__(128, 2) prefill_mma_kernel(float* __restrict__ out, const float* __restrict__ Q,
                                                             const __half* __restrict__ kc, const __half* __restrict__ vc,
                                                             int seq_len, int start_pos, int n_heads, int n_kv, int max_seq,
                                                             float scale, int window, int keep, float softcap, int maps, int chunk,
                                                             const float* __restrict__ sink, int joint_v, const float* __restrict__ slopes, float* __restrict__ parts) {
    constexpr int LD = HD + PAD, LDV = HDV + PAD, KS = HD / 16, NT = HDV / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* sK = reinterpret_cast<__half*>(smem_raw);                 // [2][BKV][LD]
    __half* sV = sK + 2 * BKV * LD;                                   // [2][BKV][LDV]
    const int qb = gridDim.x - 1 - blockIdx.x;                        // heaviest (latest) query blocks first
    const int head = blockIdx.y, vh = (head / maps) / ((n_heads / maps) / n_kv), kvh = vh * maps + head % maps, n_k = n_kv * maps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = qb * BQ + warp * 16 + g, r1 = r0 + 8;              // this thread's two query rows (chunk-relative)
    const float slope = slopes ? slopes[head / maps] : 0.f;           // slope * (p - key) is taken off the score
    const int p0 = start_pos + r0, p1 = start_pos + r1;               // their absolute positions == last visible key

    // ---- Q fragments (A operand, 16 x HD per warp), split into F16 hi + lo ----
    uint32_t qhi[KS][4], qlo[KS][4];
    float g0 = 1.f, g1 = 1.f, f0 = scale, f1 = scale;                 // SLICED: the rows' powers of two, and the scale without them
    if constexpr (SLICED) {
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int i = 0; i < KS * 2; i++) {
            const float* q = Q + ((size_t)r0 * n_heads + head) * HD + i * 8 + 2 * t;
            if (r0 < seq_len) { const float2 x = *reinterpret_cast<const float2*>(q); a0 = fmaxf(a0, fmaxf(fabsf(x.x), fabsf(x.y))); }
            if (r1 < seq_len) { const float2 x = *reinterpret_cast<const float2*>(q + (size_t)8 * n_heads * HD); a1 = fmaxf(a1, fmaxf(fabsf(x.x), fabsf(x.y))); }
        }
        auto power = [&](float amax, float& g, float& f) {
            amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1)); amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
            const uint32_t e = __float_as_uint(amax) >> 23;
            const uint32_t up = e == 255u || e == 0u ? 127u : min(227u, max(27u, 264u - e));         // to 2^10 .. 2^11; not finite, or zero: as it is
            g = __uint_as_float(up << 23); f = scale * __uint_as_float((254u - up) << 23);
        };
        power(a0, g0, f0); power(a1, g1, f1);
    }
#pragma unroll
    for (int ks = 0; ks < KS; ks++) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = (i & 1) ? r1 : r0, c = ks * 16 + 2 * t + ((i & 2) ? 8 : 0);
            float2 v = make_float2(0.f, 0.f);
            if (r < seq_len) v = *reinterpret_cast<const float2*>(Q + ((size_t)r * n_heads + head) * HD + c);
            if constexpr (SLICED) { const float x = (i & 1) ? g1 : g0; v.x *= x; v.y *= x; }
            split2<BF>(v.x, v.y, qhi[ks][i], qlo[ks][i]);
        }
    }
    float o[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

    const int last_q = min(qb * BQ + BQ, seq_len) - 1;                // last valid query of the block
    // key tiles: those of the kept prefix that lie before the block's window, then the window's (full causal: all from tile 0)
    // (chunk: from the tile holding the first row of the first query's block of positions; later queries' blocks start no earlier)
    const int first_win = chunk > 0 ? ((start_pos + qb * BQ) / chunk * chunk) / BKV : (window > 0 ? max(0, start_pos + qb * BQ - window + 1) / BKV : 0);
    const int n_keep = (window > 0 && chunk <= 0) ? min((keep + BKV - 1) / BKV, first_win) : 0;
    const int n_tiles = n_keep + (start_pos + last_q) / BKV + 1 - first_win;
    const int per = SLICED ? slice_tiles(n_tiles, gridDim.z) : n_tiles, j0 = SLICED ? blockIdx.z * per : 0, j1 = SLICED ? min(n_tiles, j0 + per) : n_tiles;
    auto tile_of = [&](int j) { return j < n_keep ? j : first_win + (j - n_keep); };

    auto load_tile = [&](int j, int st) {
        constexpr int CH = HD / 8, CHV = HDV / 8;                     // 16-byte chunks per row
        for (int c = threadIdx.x; c < BKV * CH; c += 128) {
            const int row = c / CH, ch = c % CH;
            const int key = min(tile_of(j) * BKV + row, max_seq - 1); // rows past the last are masked by causality anyway
            cp_async16(sK + ((size_t)st * BKV + row) * LD + ch * 8, kc + ((size_t)key * n_k + kvh) * HD + ch * 8);
        }
        for (int c = threadIdx.x; c < BKV * CHV; c += 128) {
            const int row = c / CHV, ch = c % CHV;
            const int key = min(tile_of(j) * BKV + row, max_seq - 1);
            cp_async16(sV + ((size_t)st * BKV + row) * LDV + ch * 8, vc + (joint_v ? (size_t)key : (size_t)key * n_kv + vh) * HDV + ch * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const bool plain = window <= 0 && chunk <= 0 && softcap <= 0.f && !slopes;
    if (!SLICED || j0 < j1) load_tile(j0, 0);
    for (int j = j0; j < j1; j++) {
        const int st = (j - j0) & 1;
        if (j + 1 < j1) {
            load_tile(j + 1, st ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const __half* tK = sK + (size_t)st * BKV * LD;
        const __half* tV = sV + (size_t)st * BKV * LDV;

        // ---- S = Q K^T (16 x 64 per warp) ----
        float s[8][4];
        if constexpr (SLICED) {
            constexpr int HALF = KS / 2;
#pragma unroll
            for (int h = 0; h < 2; h++) {                    // 32 keys at a time: four sums of high halves and four of low ones side by side
#pragma unroll
                for (int n = 0; n < 4; n++) s[4 * h + n][0] = s[4 * h + n][1] = s[4 * h + n][2] = s[4 * h + n][3] = 0.f;
                float lo[4][4] = {};
#pragma unroll
                for (int part = 0; part < 2; part++) {
                    float d[4][4] = {};
#pragma unroll
                    for (int ks = part * HALF; ks < (part + 1) * HALF; ks++) {
                        uint32_t kb[2][4];
#pragma unroll
                        for (int n2 = 0; n2 < 2; n2++) {
                            const __half* kp = tK + (size_t)((2 * h + n2) * 16 + (lane & 7) + (lane >> 4) * 8) * LD + ks * 16 + ((lane >> 3) & 1) * 8;
                            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(kb[n2][0]), "=r"(kb[n2][1]), "=r"(kb[n2][2]), "=r"(kb[n2][3]) : "r"((uint32_t)__cvta_generic_to_shared(kp)));
                        }
#pragma unroll
                        for (int n = 0; n < 4; n++) mma16816<BF>(d[n], qhi[ks], kb[n >> 1][2 * (n & 1)], kb[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
                        for (int n = 0; n < 4; n++) mma16816<BF>(lo[n], qlo[ks], kb[n >> 1][2 * (n & 1)], kb[n >> 1][2 * (n & 1) + 1]);
                    }
#pragma unroll
                    for (int n = 0; n < 4; n++)
#pragma unroll
                        for (int i = 0; i < 4; i++) s[4 * h + n][i] += d[n][i];
                }
#pragma unroll
                for (int n = 0; n < 4; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++) s[4 * h + n][i] += lo[n][i];
            }
        } else {
#pragma unroll
        for (int n = 0; n < 8; n++) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
            // all eight blocks of keys with the high half, then with the low: a product waits for the one eight before it, not for its neighbour
            uint32_t kb[4][4];
#pragma unroll
            for (int n2 = 0; n2 < 4; n2++) {             // four 8x8 blocks of K: (keys +0..7 | +8..15) x (dims +0..7 | +8..15)
                const __half* kp = tK + (size_t)(n2 * 16 + (lane & 7) + (lane >> 4) * 8) * LD + ks * 16 + ((lane >> 3) & 1) * 8;
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                             : "=r"(kb[n2][0]), "=r"(kb[n2][1]), "=r"(kb[n2][2]), "=r"(kb[n2][3]) : "r"((uint32_t)__cvta_generic_to_shared(kp)));
            }
#pragma unroll
            for (int n = 0; n < 8; n++) mma16816<BF>(s[n], qhi[ks], kb[n >> 1][2 * (n & 1)], kb[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
            for (int n = 0; n < 8; n++) mma16816<BF>(s[n], qlo[ks], kb[n >> 1][2 * (n & 1)], kb[n >> 1][2 * (n & 1) + 1]);
        }
        }
        // ---- scale, causal mask, online softmax ----
        const int key0 = tile_of(j) * BKV;
        float mx0 = -INFINITY, mx1 = -INFINITY;
        // a tile that every row of the warp sees whole, without cap or slope, needs no per-score rule
        if (plain && key0 + BKV - 1 <= start_pos + qb * BQ + warp * 16) {
#pragma unroll
            for (int n = 0; n < 8; n++) {
#pragma unroll
                for (int i = 0; i < 4; i++) s[n][i] *= (i & 2) ? f1 : f0;
                mx0 = fmaxf(mx0, fmaxf(s[n][0], s[n][1]));
                mx1 = fmaxf(mx1, fmaxf(s[n][2], s[n][3]));
            }
        } else
#pragma unroll
        for (int n = 0; n < 8; n++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int key = key0 + n * 8 + 2 * t + (i & 1);
                const int p = (i & 2) ? p1 : p0;
                const bool seen = key <= p && (chunk > 0 ? key >= p / chunk * chunk : (window <= 0 || p - key < window || key < keep));
                float v = s[n][i] * ((i & 2) ? f1 : f0);
                if (softcap > 0.f) v = softcap * (1.0f - 2.0f / (__expf(2.0f * v / softcap) + 1.0f));     // cap * tanh(v / cap)
                v -= slope * (float)(p - key);
                v = seen ? v : -INFINITY;
                s[n][i] = v;
                if (i & 2) mx1 = fmaxf(mx1, v); else mx0 = fmaxf(mx0, v);
            }
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xFFFFFFFFu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xFFFFFFFFu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xFFFFFFFFu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xFFFFFFFFu, mx1, 2));
        // full causal: finite from tile 0 on (key 0 is visible to every row); with a window a row can find a whole tile masked
        // before its first visible key: subtract 0 instead of -inf so every exponential is exp(-inf) = 0, not NaN
        const float mr0 = fmaxf(m0, mx0), mr1 = fmaxf(m1, mx1);
        const float mn0 = mr0 == -INFINITY ? 0.f : mr0, mn1 = mr1 == -INFINITY ? 0.f : mr1;
        const float a0 = __expf(m0 - mn0), a1 = __expf(m1 - mn1);
        m0 = mr0; m1 = mr1;
        float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
        for (int n = 0; n < 8; n++) {
            s[n][0] = __expf(s[n][0] - mn0); s[n][1] = __expf(s[n][1] - mn0);
            s[n][2] = __expf(s[n][2] - mn1); s[n][3] = __expf(s[n][3] - mn1);
            sum0 += s[n][0] + s[n][1]; sum1 += s[n][2] + s[n][3];
        }
        l0 = l0 * a0 + sum0; l1 = l1 * a1 + sum1;                    // per-thread partial row sums (reduced at the end)
        if constexpr (SLICED) {
            uint32_t phi[BKV / 16][4], plo[BKV / 16][4];
#pragma unroll
            for (int kt = 0; kt < BKV / 16; kt++)
#pragma unroll
                for (int i = 0; i < 4; i++) split2<BF>(s[2 * kt + (i >> 1)][2 * (i & 1)], s[2 * kt + (i >> 1)][2 * (i & 1) + 1], phi[kt][i], plo[kt][i]);
            constexpr int G = 4;                                         // blocks of 16 columns at a time
#pragma unroll
            for (int np = 0; np < HDV / 16; np += G) {
                float d[2 * G][4];
#pragma unroll
                for (int n = 0; n < 2 * G; n++) d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0.f;
#pragma unroll
                for (int kt = 0; kt < BKV / 16; kt++) {
                    uint32_t v[G][4];
#pragma unroll
                    for (int q = 0; q < G; q++) {
                        const __half* vp = tV + (size_t)(kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDV + (np + q) * 16 + (lane >> 4) * 8;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(v[q][0]), "=r"(v[q][1]), "=r"(v[q][2]), "=r"(v[q][3]) : "r"((uint32_t)__cvta_generic_to_shared(vp)));
                    }
#pragma unroll
                    for (int q = 0; q < G; q++) { mma16816<BF>(d[2 * q], plo[kt], v[q][0], v[q][1]); mma16816<BF>(d[2 * q + 1], plo[kt], v[q][2], v[q][3]); }
#pragma unroll
                    for (int q = 0; q < G; q++) { mma16816<BF>(d[2 * q], phi[kt], v[q][0], v[q][1]); mma16816<BF>(d[2 * q + 1], phi[kt], v[q][2], v[q][3]); }
                }
#pragma unroll
                for (int n = 0; n < 2 * G; n++) {
                    float (&x)[4] = o[2 * np + n];
                    x[0] = fmaf(x[0], a0, d[n][0]); x[1] = fmaf(x[1], a0, d[n][1]); x[2] = fmaf(x[2], a1, d[n][2]); x[3] = fmaf(x[3], a1, d[n][3]);
                }
            }
            __syncthreads();
            continue;
        }
#pragma unroll
        for (int n = 0; n < NT; n++) { o[n][0] *= a0; o[n][1] *= a0; o[n][2] *= a1; o[n][3] *= a1; }

        // ---- O += P V : the accumulator layout of S is the A-operand layout of the second MMA ----
#pragma unroll
        for (int kt = 0; kt < BKV / 16; kt++) {
            uint32_t phi[4], plo[4];
            split2<BF>(s[2 * kt][0], s[2 * kt][1], phi[0], plo[0]);
            split2<BF>(s[2 * kt][2], s[2 * kt][3], phi[1], plo[1]);
            split2<BF>(s[2 * kt + 1][0], s[2 * kt + 1][1], phi[2], plo[2]);
            split2<BF>(s[2 * kt + 1][2], s[2 * kt + 1][3], phi[3], plo[3]);
            constexpr int G = HDV % 64 == 0 ? 4 : HDV % 32 == 0 ? 2 : 1;     // blocks of 16 columns whose products are interleaved
#pragma unroll
            for (int np = 0; np < HDV / 16; np += G) {
                // four 8x8 blocks of V^T: (keys +0..7 | +8..15) x (hd +0..7 | +8..15)
                uint32_t v[G][4];
#pragma unroll
                for (int q = 0; q < G; q++) {
                    const __half* vp = tV + (size_t)(kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDV + (np + q) * 16 + (lane >> 4) * 8;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(v[q][0]), "=r"(v[q][1]), "=r"(v[q][2]), "=r"(v[q][3]) : "r"((uint32_t)__cvta_generic_to_shared(vp)));
                }
#pragma unroll
                for (int q = 0; q < G; q++) { mma16816<BF>(o[2 * (np + q)], phi, v[q][0], v[q][1]); mma16816<BF>(o[2 * (np + q) + 1], phi, v[q][2], v[q][3]); }
#pragma unroll
                for (int q = 0; q < G; q++) { mma16816<BF>(o[2 * (np + q)], plo, v[q][0], v[q][1]); mma16816<BF>(o[2 * (np + q) + 1], plo, v[q][2], v[q][3]); }
            }
        }
        __syncthreads();                                             // this stage is overwritten by the prefetch of tile j + 2
    }
    l0 += __shfl_xor_sync(0xFFFFFFFFu, l0, 1); l0 += __shfl_xor_sync(0xFFFFFFFFu, l0, 2);
    l1 += __shfl_xor_sync(0xFFFFFFFFu, l1, 1); l1 += __shfl_xor_sync(0xFFFFFFFFu, l1, 2);
    if (sink) {                     // exp(sink) joins the denominator; the maximum is raised to the sink first so nothing overflows
        const float sk = sink[head / maps];
        const float n0 = fmaxf(m0, sk), n1 = fmaxf(m1, sk);
        const float f0 = __expf(m0 - n0), f1 = __expf(m1 - n1);
        l0 = l0 * f0 + __expf(sk - n0); l1 = l1 * f1 + __expf(sk - n1);
#pragma unroll
        for (int n = 0; n < NT; n++) { o[n][0] *= f0; o[n][1] *= f0; o[n][2] *= f1; o[n][3] *= f1; }
    }
    if constexpr (SLICED) {
        float2* ml = reinterpret_cast<float2*>(parts + (size_t)gridDim.z * seq_len * n_heads * HDV);
        const size_t at0 = ((size_t)blockIdx.z * seq_len + r0) * n_heads + head, at1 = at0 + (size_t)8 * n_heads;
        if (t == 0 && r0 < seq_len) ml[at0] = make_float2(m0, l0);
        if (t == 0 && r1 < seq_len) ml[at1] = make_float2(m1, l1);
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const int c = n * 8 + 2 * t;
            if (r0 < seq_len) *reinterpret_cast<float2*>(parts + at0 * HDV + c) = make_float2(o[n][0], o[n][1]);
            if (r1 < seq_len) *reinterpret_cast<float2*>(parts + at1 * HDV + c) = make_float2(o[n][2], o[n][3]);
        }
        return;
    }
    const float i0 = 1.0f / l0, i1 = 1.0f / l1;
#pragma unroll
    for (int n = 0; n < NT; n++) {
        const int c = n * 8 + 2 * t;
        if (r0 < seq_len) *reinterpret_cast<float2*>(out + ((size_t)r0 * n_heads + head) * HDV + c) = make_float2(o[n][0] * i0, o[n][1] * i0);
        if (r1 < seq_len) *reinterpret_cast<float2*>(out + ((size_t)r1 * n_heads + head) * HDV + c) = make_float2(o[n][2] * i1, o[n][3] * i1);
    }
}

// A warp to a query's head: sum_i e^{m_i - m} o_i / sum_i e^{m_i - m} l_i over the slices.  All latency: whatever it reads is fetched at once.
constexpr int SLICES = 16;
struct MergeAttn {
    float* out;
    const float *Q, *parts;
    const __half *kc, *vc;
    int rows, slices, start_pos, n_heads, n_kv;
    float scale;
};
template <int HD>
__global__ void __launch_bounds__(128) prefill_merge_kernel(const __grid_constant__ MergeAttn p) {
    constexpr int C = HD / 32;
    pdl_launch_dependents();
    pdl_wait();
    const float* parts = behind_wait(p.parts);
    const int at = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;      // (query, head)
    if (at >= p.rows) return;
    const float2* ml = reinterpret_cast<const float2*>(parts + (size_t)p.slices * p.rows * HD);
    // Slices that begin behind the query's position are left out, and no others: a weight of zero is none of a NaN or infinite sum of values that the query sees
    const int row = at / p.n_heads, last = min(row / BQ * BQ + BQ, p.rows / p.n_heads) - 1;
    const int seen = (p.start_pos + row) / BKV / slice_tiles((p.start_pos + last) / BKV + 1, p.slices) + 1;
    float2 mine = make_float2(-INFINITY, 0.f);
    if (lane < p.slices) mine = ml[(size_t)lane * p.rows + at];
    float o[SLICES][C];
#pragma unroll
    for (int i = 0; i < SLICES; i++)
#pragma unroll
        for (int c = 0; c < C; c++) o[i][c] = i < p.slices ? parts[((size_t)i * p.rows + at) * HD + lane * C + c] : 0.f;
    float m = mine.x;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, d));
    const float w = __expf(mine.x - m);
    float l = lane < seen ? w * mine.y : 0.f, sum[C] = {};
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, d);
    float odd = 0.f;                                          // NaN where a sum is infinite or NaN
#pragma unroll
    for (int i = 0; i < SLICES; i++) {
        const float wi = __shfl_sync(0xFFFFFFFFu, w, i);
        if (i < seen)
#pragma unroll
            for (int c = 0; c < C; c++) sum[c] = fmaf(o[i][c], wi, sum[c]);
    }
    const float inv = 1.0f / l;
#pragma unroll
    for (int c = 0; c < C; c++) {
        odd = fmaf(sum[c], 0.f, odd);
        p.out[(size_t)at * HD + lane * C + c] = sum[c] * inv;
    }
    if (__any_sync(0xFFFFFFFFu, !(odd == 0.f)) && l < INFINITY) row_alone<HD, HD>(p, at / p.n_heads, at % p.n_heads, 0, lane);      // (a row that sees a NaN or infinite score is NaN)
}

template <int HD, int HDV, bool BF, bool SLICED = false>
void launch(float* out, const float* Q, const __half* kc, const __half* vc, int seq_len, int start_pos, int n_heads, int n_kv,
            int max_seq, float scale, int window, int keep, float softcap, cudaStream_t s, int maps = 1, int chunk = 0, const float* sink = nullptr,
            int joint_v = 0, const float* slopes = nullptr, float* parts = nullptr, int slices = 1) {
    const int smem = 2 * BKV * (HD + PAD + HDV + PAD) * (int)sizeof(__half);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(prefill_mma_kernel<HD, HDV, BF, SLICED>, (int)(smem), configured);
    // The cache ends with the last query for it: what lies behind may be infinite or NaN, and a masked row's weight of zero times that would be NaN.
    max_seq = std::min(max_seq, std::max(1, start_pos + seq_len));
    // (not programmatic: CTAs that wait for the launch before would gather two to an SM where it is done; 64 heads, 128 tokens behind 4000: 131 us, 206)
    prefill_mma_kernel<HD, HDV, BF, SLICED><<<dim3((seq_len + BQ - 1) / BQ, n_heads * maps, slices), 128, smem, s>>>(out, Q, kc, vc, seq_len, start_pos, n_heads * maps, n_kv,
                                                                                                    max_seq, scale, window, keep, softcap, maps, chunk, sink, joint_v, slopes, parts);
    NT_LAUNCH_CHECK();
    count_launch();
}

}  // namespace

bool attention_prefill_mma_supported(int seq_len, int n_heads, int n_kv, int hd) {
    return seq_len >= 16 && (hd == 64 || hd == 128) && n_kv > 0 && n_heads % n_kv == 0;
}

void attention_prefill_mma(float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads,
                           int n_kv, int hd, int max_seq, float scale, cudaStream_t s) {
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
    if (hd == 128) launch<128, 128, false>(out, Q, k, v, seq_len, start_pos, n_heads, n_kv, max_seq, scale, 0, 0, 0.f, s);
    else launch<64, 64, false>(out, Q, k, v, seq_len, start_pos, n_heads, n_kv, max_seq, scale, 0, 0, 0.f, s);
}

// The keys in slices, each with CTAs of its own, and a merge: for few CTAs that walk many keys.  false: no memory, nothing launched
bool attention_prefill_slices(float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads, int n_kv, int hd, int max_seq, float scale,
                              int slices, cudaStream_t s) {
    if (slices < 2 || slices > SLICES || (hd != 64 && hd != 128)) return false;
    const size_t rows = (size_t)seq_len * n_heads;
    StreamMemory memory(slices * rows * (hd + 2) * sizeof(float), s);
    if (!memory.p) return false;
    float* parts = static_cast<float*>(memory.p);
    const __half *k = static_cast<const __half*>(kc), *v = static_cast<const __half*>(vc);
    const dim3 grid((unsigned)((rows + 3) / 4)), block(128);
    const MergeAttn p{out, Q, parts, k, v, (int)rows, slices, start_pos, n_heads, n_kv, scale};
    if (hd == 128) {
        launch<128, 128, false, true>(out, Q, k, v, seq_len, start_pos, n_heads, n_kv, max_seq, scale, 0, 0, 0.f, s, 1, 0, nullptr, 0, nullptr, parts, slices);
        launch_k_pdl(true, prefill_merge_kernel<128>, grid, block, 0, s, p);
    } else {
        launch<64, 64, false, true>(out, Q, k, v, seq_len, start_pos, n_heads, n_kv, max_seq, scale, 0, 0, 0.f, s, 1, 0, nullptr, 0, nullptr, parts, slices);
        launch_k_pdl(true, prefill_merge_kernel<64>, grid, block, 0, s, p);
    }
    count_launch();
    return true;
}

// Windowed / block-masked / soft-capped / distance-biased form over a BF16 cache: (dim, vdim) in {(64, 64), (96, 96), (128, 128), (32, 64), (64, 128)}, one or
// two score maps per head, at least 16 queries.
bool attention_window_mma_supported(int tokens, const WindowAttn& a, DType cache_dt) {
    const bool shape = (a.dim == a.vdim && (a.dim == 64 || a.dim == 96 || a.dim == 128)) || (a.vdim == 2 * a.dim && (a.dim == 32 || a.dim == 64));
    // joint values: one value row of width vdim per key, packed (the stride equals the width)
    const bool strides = a.k_stride == 0 && (a.joint_v ? (a.v_stride == a.vdim && a.maps == 1) : a.v_stride == 0);
    return cache_dt == DType::BF16 && shape && strides && !a.head_gate && a.maps >= 1 && a.maps <= 2 && tokens >= 16 && a.kv_heads > 0 && a.heads % a.kv_heads == 0;
}
void attention_window_mma(float* out, const float* Q, const void* kc, const void* vc, int tokens, int p0, int max_seq, const WindowAttn& a,
                          cudaStream_t s) {
    const __half* k = static_cast<const __half*>(kc);       // 16-bit words either way; the BF instantiation reads them as BF16
    const __half* v = static_cast<const __half*>(vc);
#define NT_AW(D, V) launch<D, V, true>(out, Q, k, v, tokens, p0, a.heads, a.kv_heads, max_seq, a.scale, a.window, a.keep, a.softcap, s, a.maps, a.chunk, a.sink, a.joint_v, a.slope)
    if (a.dim == 128) NT_AW(128, 128);
    else if (a.dim == 96) NT_AW(96, 96);
    else if (a.dim == 64 && a.vdim == 64) NT_AW(64, 64);
    else if (a.dim == 64) NT_AW(64, 128);
    else NT_AW(32, 64);
#undef NT_AW
}

// Per-head 16-bit operands built for the call (latent attention's expanded keys / values): key width 64, 128 or 192, value width 64
// or 128, every head its own key / value head, causal or windowed mask.
bool attention_heads_mma_widths(int key_dim, int value_dim, int* kw, int* vw) {
    if (key_dim <= 0 || value_dim <= 0 || key_dim > 192 || value_dim > 128) return false;
    *kw = key_dim <= 64 ? 64 : key_dim <= 128 ? 128 : 192;
    *vw = value_dim <= 64 ? 64 : 128;
    return true;
}
void attention_heads_mma(float* out, const float* Q, const void* kc, const void* vc, int tokens, int p0, int rows, int heads, int kw, int vw, float scale,
                         cudaStream_t s, int window) {
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
#define NT_AH(D, V) launch<D, V, true>(out, Q, k, v, tokens, p0, heads, heads, rows, scale, window, 0, 0.f, s)
    if (kw == 64 && vw == 64) NT_AH(64, 64);
    else if (kw == 64 && vw == 128) NT_AH(64, 128);
    else if (kw == 128 && vw == 64) NT_AH(128, 64);
    else if (kw == 128 && vw == 128) NT_AH(128, 128);
    else if (kw == 192 && vw == 64) NT_AH(192, 64);
    else if (kw == 192 && vw == 128) NT_AH(192, 128);
    else NT_CHECK(false, "attention_heads_mma: widths from attention_heads_mma_widths");
#undef NT_AH
}

}}  // namespace nt::b200
