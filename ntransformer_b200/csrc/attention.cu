// attention.cu — GQA KV-cache attention for decode and prefill on sm_100a.
//
// Replaces reference kernels K16 (attention_decode_generic_kernel, src/cuda/attention.cu:108-202) and
// K18 (attention_prefill_kernel, :216-311).  Same math (F32 q, F16 K/V, scores * scale, softmax with the
// fast-math exp, P.V in F32) with a different work split:
//   * one CTA serves GC query heads that share a KV head, so K/V rows are fetched once per GQA group
//     instead of once per head (the reference re-reads them n_heads/n_kv_heads times);
//   * decode is split along the context (flash-decoding): grid = head-groups x splits so 148 SMs are
//     busy at ctx 2048 where the reference launches only n_heads CTAs; partial (max, sum, P.V) are merged
//     by a small combine kernel;
//   * K rows are read coalesced (one row per warp step, DPL dims per lane) and the GC partial dot
//     products are reduced with a transpose-reduce (GC-1 + log2(32/GC) shuffles instead of 5*GC).
// Compiled with --use_fast_math (expf -> ex2.approx path, as the reference build).
#include "kernels_internal.h"
#include "ring.cuh"
#include "xquant.cuh"
#include "attention_walk.cuh"
#include <cuda_fp16.h>
#include <algorithm>
#include <cfloat>
#include <optional>

namespace nt { namespace b200 {

namespace {

constexpr int AW = WALK_WARPS;           // warps per CTA
constexpr int MAX_SPLITS = 64;
// Graph-replayed decode (launch shape fixed by max_seq): a context slice holds at least this many keys.  Without the floor a short
// context is cut into one-key slices (ctx 64 over 64 slices when a rank holds a single KV head) and the merge walks them all:
// decode_combine took 13.9 us at tensor-parallel-8 shapes and 5.4 us at one GPU (profiles/r02_launches_tp8_shard.txt).
constexpr int DYN_MIN_SPLIT = 32;
constexpr int FUSED_MIN_SPLIT = 64;      // decode_fused_kernel: at least this many keys per context slice (one slice = no merge step)
constexpr int ATTN_MAX_DYN_SMEM = 227 * 1024 - 1024;   // static __shared__ counts against the 227 KB cap

// Decode-step fusion (decode_fused_kernel): the token at cache row `pos` is not in the cache yet.  Its key arrives unrotated
// in F32 from the q/k/v GEMV; the warp that reaches row `pos` rotates it (reference rotary.cu:16-62, pairs (i, i + hd/2)), rounds
// key and value to F16 exactly as the cache write does (attention.cu:338-339) and — in the one CTA per KV head that owns the
// write — stores the row.  attend_group without NEW: plain attention over the cache, queries used as given.
struct NewToken {
    const float* k = nullptr;      // [n_kv][HD]
    const float* v = nullptr;
    int pos = -1;
    float theta = 0.f, freq_scale = 1.f;
    __half* kc_w = nullptr;        // cache base pointers, non-null only in the CTA that stores the row
    __half* vc_w = nullptr;
};

// cos / sin of this lane's DPL rotation pairs.  Lane L holds dims [L*DPL, L*DPL + DPL): lanes 0-15 the first half of the
// head, lanes 16-31 the second, so a pair (i, i + hd/2) lives in lanes (L, L ^ 16) at the same register index.
// Same expression as rope_kv_decode_kernel / the reference (fast-math powf, cosf, sinf).
template <int DPL>
__device__ __forceinline__ void rope_angles(float (&c)[DPL], float (&sn)[DPL], int lane, int pos, float theta_base, float freq_scale) {
    constexpr int head_dim = DPL * 32;
#pragma unroll
    for (int i = 0; i < DPL; i++) {
        const int pair = (lane & 15) * DPL + i;
        float freq = 1.0f / powf(theta_base, (2.0f * pair) / head_dim);
        float angle = pos * freq * freq_scale;
        c[i] = cosf(angle); sn[i] = sinf(angle);
    }
}
template <int DPL>
__device__ __forceinline__ void rope_rotate(float (&x)[DPL], const float (&c)[DPL], const float (&sn)[DPL], int lane) {
#pragma unroll
    for (int i = 0; i < DPL; i++) {
        const float other = __shfl_xor_sync(0xFFFFFFFFu, x[i], 16);
        const bool lo = lane < 16;
        const float x0 = lo ? x[i] : other, x1 = lo ? other : x[i];
        const float r0 = x0 * c[i] - x1 * sn[i], r1 = x1 * c[i] + x0 * sn[i];
        x[i] = lo ? r0 : r1;
    }
}
template <int DPL>
__device__ __forceinline__ void store_row_f16(__half* p, const __half (&h)[DPL]) {
    typename HalfVec<DPL>::T raw;
    __half* d = reinterpret_cast<__half*>(&raw);
#pragma unroll
    for (int i = 0; i < DPL; i++) d[i] = h[i];
    *reinterpret_cast<typename HalfVec<DPL>::T*>(p) = raw;
}

// One CTA: GC query heads of one KV head, keys [k_begin, k_end) (attention_walk.cuh).
// q_base: first of the GC heads' query vectors (contiguous [GC][hd]); out likewise.
// If part_* != nullptr writes unnormalised partials, else the normalised output.
template <int DPL, int GC, bool NEW = false, bool APART = true>
__device__ void attend_group(float* __restrict__ out, const float* __restrict__ q_base, const __half* __restrict__ kc,
                             const __half* __restrict__ vc, int kv_head, int n_kv, int k_begin, int k_end, float scale,
                             float* __restrict__ part_o, float* __restrict__ part_ml, float* smem, const NewToken nt = NewToken{}) {
    constexpr int HD = DPL * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t row_stride = (size_t)n_kv * HD, channel = (size_t)kv_head * HD + (size_t)lane * DPL;
    float rc[DPL], rs[DPL];
    walk_slice<DPL, GC, NEW, APART>(kc + channel, vc + channel, row_stride, k_begin, k_end, nt.pos, scale, smem, warp, lane,
        [&](float (&qr)[GC][DPL]) {
#pragma unroll
            for (int g = 0; g < GC; g++)
#pragma unroll
                for (int i = 0; i < DPL; i++) qr[g][i] = q_base[(size_t)g * HD + lane * DPL + i];
            if (NEW) {                                   // fused decode step: the queries arrive unrotated
                rope_angles<DPL>(rc, rs, lane, nt.pos, nt.theta, nt.freq_scale);
#pragma unroll
                for (int g = 0; g < GC; g++) rope_rotate<DPL>(qr[g], rc, rs, lane);
            }
        },
        [&](float (&kf)[DPL]) {                          // the new token's key, not in the cache yet
#pragma unroll
            for (int i = 0; i < DPL; i++) kf[i] = nt.k[(size_t)kv_head * HD + lane * DPL + i];
            rope_rotate<DPL>(kf, rc, rs, lane);
            __half kh[DPL];
#pragma unroll
            for (int i = 0; i < DPL; i++) { kh[i] = __float2half(kf[i]); kf[i] = __half2float(kh[i]); }
            if (nt.kc_w) store_row_f16<DPL>(nt.kc_w + (size_t)nt.pos * row_stride + channel, kh);
        },
        [&](float (&vf)[DPL]) {                          // the new token's value: F16-rounded like the cache row it becomes
            __half vh[DPL];
#pragma unroll
            for (int i = 0; i < DPL; i++) { vh[i] = __float2half(nt.v[(size_t)kv_head * HD + lane * DPL + i]); vf[i] = __half2float(vh[i]); }
            if (nt.vc_w) store_row_f16<DPL>(nt.vc_w + (size_t)nt.pos * row_stride + channel, vh);
        });
    __syncthreads();
    for (int idx = threadIdx.x; idx < GC * HD; idx += AW * 32) {
        const int g = idx / HD, d = idx - g * HD;
        float m, l, t;
        walk_merge<DPL, GC>(smem, idx, m, l, t);
        if (part_o) {
            part_o[(size_t)g * HD + d] = t;             // caller strides heads by HD inside its split slot
            if (d == 0) { part_ml[2 * g] = m; part_ml[2 * g + 1] = l; }
        } else {
            out[(size_t)g * HD + d] = t * ((l > 0.f) ? 1.0f / l : 0.f);
        }
    }
}

// Scratch layout for split decode: [head][split][HD] floats then [head][split][2] (max, sum).
template <int DPL, int GC, bool APART = true>
__global__ void __launch_bounds__(AW * 32, DPL * GC <= 32 ? 2 : 1) decode_kernel(float* __restrict__ out, const float* __restrict__ q,
                                                         const __half* __restrict__ kc, const __half* __restrict__ vc,
                                                         int seq_len, int n_heads, int n_kv, float scale, int n_splits,
                                                         int split_len, float* __restrict__ scratch,
                                                         const int* __restrict__ pos_dev) {
    constexpr int HD = DPL * 32;
    extern __shared__ float smem_dyn[];
    pdl_wait();
    pdl_launch_dependents();
    q = behind_wait(q); kc = behind_wait(kc); vc = behind_wait(vc); pos_dev = behind_wait(pos_dev);
    if (pos_dev) {                       // CUDA-graph replay: context length lives in device memory
        seq_len = *pos_dev + 1;
        split_len = max((seq_len + n_splits - 1) / n_splits, DYN_MIN_SPLIT);
    }
    if (blockIdx.z) {                    // a run of tokens: query z attends one key more than the one before it (slices cut for the last)
        seq_len += blockIdx.z;
        q += (size_t)blockIdx.z * n_heads * HD;
        out += (size_t)blockIdx.z * n_heads * HD;
        scratch += (size_t)blockIdx.z * n_heads * n_splits * (HD + 2);
    }
    const int head0 = blockIdx.x * GC, split = blockIdx.y;
    const int kv_head = head0 / (n_heads / n_kv);
    const int k_begin = split * split_len, k_end = min(seq_len, k_begin + split_len);
    if (k_begin >= k_end) return;
    if (n_splits == 1 && !pos_dev) {
        attend_group<DPL, GC, false, APART>(out + (size_t)head0 * HD, q + (size_t)head0 * HD, kc, vc, kv_head, n_kv, k_begin, k_end, scale,
                              nullptr, nullptr, smem_dyn);
    } else {
        // partials for head (head0+g) live at scratch[((head0+g) * n_splits + split) * HD]; attend_group strides
        // heads by HD, so hand it a staging area in shared memory and scatter afterwards.
        float* stage = smem_dyn + walk_floats<DPL, GC>();   // [GC][HD] + [GC][2]
        attend_group<DPL, GC, false, APART>(nullptr, q + (size_t)head0 * HD, kc, vc, kv_head, n_kv, k_begin, k_end, scale, stage,
                              stage + GC * HD, smem_dyn);
        __syncthreads();
        float* ml = scratch + (size_t)n_heads * n_splits * HD;
        for (int idx = threadIdx.x; idx < GC * HD; idx += AW * 32) {
            const int g = idx / HD, d = idx - g * HD;
            scratch[((size_t)(head0 + g) * n_splits + split) * HD + d] = stage[idx];
        }
        if (threadIdx.x < 2 * GC) {
            const int g = threadIdx.x >> 1;
            ml[((size_t)(head0 + g) * n_splits + split) * 2 + (threadIdx.x & 1)] = stage[GC * HD + threadIdx.x];
        }
    }
}

// Merge split partials: out[h] = sum_i e^{m_i - m} o_i / sum_i e^{m_i - m} l_i
// xq_out (optional): also emits the block-scaled int8x3 form of the output vector (kernels_internal.h "xq") that
// the o-projection GEMV consumes, saving a separate quantise launch.  Requires blockDim.x == 128, hd % 32 == 0.
__global__ void __launch_bounds__(128) decode_combine_kernel(float* __restrict__ out, const float* __restrict__ scratch, int n_heads, int hd,
                                      int n_splits, int seq_len, int split_len, const int* __restrict__ pos_dev,
                                      int8_t* __restrict__ xq_out) {
    __shared__ float w_s[MAX_SPLITS];                // e^{m_i - m} per slice
    __shared__ float inv_s;
    const int h = blockIdx.x;
    pdl_wait();
    pdl_launch_dependents();
    scratch = behind_wait(scratch); pos_dev = behind_wait(pos_dev);
    seq_len += blockIdx.y;               // a run of tokens: blockIdx.y is the query
    scratch += (size_t)blockIdx.y * n_heads * n_splits * (hd + 2);
    out += (size_t)blockIdx.y * n_heads * hd;
    if (pos_dev) { seq_len = *pos_dev + 1; split_len = max((seq_len + n_splits - 1) / n_splits, DYN_MIN_SPLIT); }
    const float* ml = scratch + (size_t)n_heads * n_splits * hd + (size_t)h * n_splits * 2;
    const int used = (seq_len + split_len - 1) / split_len;
    // All latency: everything the merge reads is fetched at once, the slices' (max, sum) pairs by the first warp (a lane has slices lane and lane + 32) and a channel
    // of every slice by each thread.  64 heads, 4000 keys: 14.5 -> 12.3 us for slices and merge, where a channel's slices came eight at a time behind the weights.
    const bool first = threadIdx.x < 32;
    const int i0 = threadIdx.x, i1 = threadIdx.x + 32;
    float m0 = -FLT_MAX, l0 = 0.f, m1 = -FLT_MAX, l1 = 0.f;
    if (first && i0 < used) { m0 = ml[2 * i0]; l0 = ml[2 * i0 + 1]; }
    if (first && i1 < used) { m1 = ml[2 * i1]; l1 = ml[2 * i1 + 1]; }
    float t[MAX_SPLITS];
    auto fetch = [&](int d) {
        const float* sp = scratch + (size_t)h * n_splits * hd + d;
#pragma unroll
        for (int c = 0; c < MAX_SPLITS; c += 16) {
            if (c >= used) break;
#pragma unroll
            for (int j = 0; j < 16; j++) t[c + j] = c + j < used ? sp[(size_t)(c + j) * hd] : 0.f;
        }
    };
    if (threadIdx.x < hd) fetch(threadIdx.x);
    if (first) {
        float m = fmaxf(m0, m1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        const float w0 = (i0 < used) ? expf(m0 - m) : 0.f, w1 = (i1 < used) ? expf(m1 - m) : 0.f;
        float l = l0 * w0 + l1 * w1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
        w_s[i0] = w0;
        w_s[i1] = w1;
        if (threadIdx.x == 0) inv_s = (l > 0.f) ? 1.0f / l : 0.f;
    }
    __syncthreads();
    const float inv = inv_s;
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {       // hd % 32 == 0: whole warps stay together
        if (d >= (int)blockDim.x) fetch(d);
        float o = 0.f;
#pragma unroll
        for (int c = 0; c < MAX_SPLITS; c += 16) {
            if (c >= used) break;
#pragma unroll
            for (int j = 0; j < 16; j++) o = c + j < used ? fmaf(t[c + j], w_s[c + j], o) : o;
        }
        const float v = o * inv;
        out[(size_t)h * hd + d] = v;
        if (xq_out) {
            const int K = n_heads * hd, e = h * hd + d, lane = threadIdx.x & 31;
            int q1, q2, q3;
            float sc, s16;
            quantize_lane32(v, q1, q2, q3, sc, s16);
            const int se = (int)xq_swizzle((uint32_t)e);
            xq_out[se] = (int8_t)q1;
            xq_out[K + se] = (int8_t)q2;
            xq_out[2 * K + se] = (int8_t)q3;
            float* scale = reinterpret_cast<float*>(xq_out + 3 * (size_t)K);
            if (lane == 0) scale[e >> 5] = sc;
            if ((lane & 15) == 0) scale[K / 32 + (e >> 4)] = s16;
        }
    }
}

// The decode step's whole attention sub-block in ONE launch: RoPE of the queries and of the new key, the F16 KV-cache write
// at row *pos_dev, split-context GQA attention, and — by the CTA that finishes a head group's last split ("last arriver", one
// ticket per head group) — the merge of the splits and the xq form of the result for the o-projection.  Replaces
// rope_kv_decode_kernel + decode_kernel + decode_combine_kernel (reference K14 rotary.cu:16-62, K15 attention.cu:316-342,
// K16 attention.cu:108-202); the merge keeps decode_combine_kernel's arithmetic and order, so both paths agree bit for bit
// whenever they cut the context at the same places.
template <int DPL, int GC>
__global__ void __launch_bounds__(AW * 32, DPL * GC <= 32 ? 2 : 1) decode_fused_kernel(float* __restrict__ out, const float* __restrict__ q,
                                                               const float* __restrict__ k_new, const float* __restrict__ v_new,
                                                               __half* __restrict__ kc, __half* __restrict__ vc,
                                                               const int* __restrict__ pos_dev, int n_heads, int n_kv, float scale,
                                                               float theta, float freq_scale, int n_splits, int min_split,
                                                               float* __restrict__ scratch, unsigned* __restrict__ tickets,
                                                               int8_t* __restrict__ xq_out) {
    constexpr int HD = DPL * 32;
    extern __shared__ float smem_dyn[];
    __shared__ int s_last;
    pdl_wait();
    pdl_launch_dependents();
    const int pos = *pos_dev, seq_len = pos + 1;
    int split_len = (seq_len + n_splits - 1) / n_splits;
    if (split_len < min_split) split_len = min_split;      // short contexts: few, reasonably long slices
    const int used = (seq_len + split_len - 1) / split_len;
    const int head0 = blockIdx.x * GC, split = blockIdx.y;
    const int per_kv = n_heads / n_kv, kv_head = head0 / per_kv;
    const int k_begin = split * split_len, k_end = min(seq_len, k_begin + split_len);
    if (k_begin >= k_end) return;
    NewToken nt;
    nt.k = k_new; nt.v = v_new; nt.pos = pos; nt.theta = theta; nt.freq_scale = freq_scale;
    if (head0 % per_kv == 0) { nt.kc_w = kc; nt.vc_w = vc; }      // one CTA per KV head stores the new row (the split that holds pos)
    if (used == 1 && !xq_out && tickets) {                 // short context: one slice per head group, normalised output, no merge
        attend_group<DPL, GC, true>(out + (size_t)head0 * HD, q + (size_t)head0 * HD, kc, vc, kv_head, n_kv, k_begin, k_end, scale, nullptr, nullptr,
                              smem_dyn, nt);
        return;
    }
    float* stage = smem_dyn + walk_floats<DPL, GC>();   // [GC][HD] + [GC][2]
    attend_group<DPL, GC, true>(nullptr, q + (size_t)head0 * HD, kc, vc, kv_head, n_kv, k_begin, k_end, scale, stage, stage + GC * HD,
                          smem_dyn, nt);
    __syncthreads();
    float* ml_all = scratch + (size_t)n_heads * n_splits * HD;
    for (int idx = threadIdx.x; idx < GC * HD; idx += AW * 32) {
        const int g = idx / HD, d = idx - g * HD;
        scratch[((size_t)(head0 + g) * n_splits + split) * HD + d] = stage[idx];
    }
    if (threadIdx.x < 2 * GC) {
        const int g = threadIdx.x >> 1;
        ml_all[((size_t)(head0 + g) * n_splits + split) * 2 + (threadIdx.x & 1)] = stage[GC * HD + threadIdx.x];
    }
    if (!tickets) return;                                  // two-launch form: decode_combine_kernel merges (attention_decode_rope_dyn)
    // ---- last arriver of the head group merges the splits ----
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned prev = atomicAdd(tickets + blockIdx.x, 1u);
        s_last = ((int)prev + 1 == used);
        if (s_last) tickets[blockIdx.x] = 0;                   // ready for the next launch (all arrivals are in)
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int g = warp; g < GC; g += AW) {
        const int h = head0 + g;
        const float* ml = ml_all + (size_t)h * n_splits * 2;
        float m = -FLT_MAX;
        for (int i = 0; i < used; i++) m = fmaxf(m, __ldcg(ml + 2 * i));
        float l = 0.f;
        for (int i = 0; i < used; i++) l += __ldcg(ml + 2 * i + 1) * expf(__ldcg(ml + 2 * i) - m);
        const float inv = (l > 0.f) ? 1.0f / l : 0.f;
        for (int d = lane; d < HD; d += 32) {
            float o = 0.f;
            for (int i = 0; i < used; i++) o += __ldcg(scratch + ((size_t)h * n_splits + i) * HD + d) * expf(__ldcg(ml + 2 * i) - m);
            const float v = o * inv;
            out[(size_t)h * HD + d] = v;
            if (xq_out) {
                const int K = n_heads * HD, e = h * HD + d;
                int q1, q2, q3;
                float sc, s16;
                quantize_lane32(v, q1, q2, q3, sc, s16);
                const int se = (int)xq_swizzle((uint32_t)e);
                xq_out[se] = (int8_t)q1;
                xq_out[K + se] = (int8_t)q2;
                xq_out[2 * K + se] = (int8_t)q3;
                float* xscale = reinterpret_cast<float*>(xq_out + 3 * (size_t)K);
                if (lane == 0) xscale[e >> 5] = sc;
                if ((lane & 15) == 0) xscale[K / 32 + (e >> 4)] = s16;
            }
        }
    }
}

template <int DPL, int GC>
__global__ void __launch_bounds__(AW * 32, DPL * GC <= 32 ? 2 : 1) prefill_kernel(float* __restrict__ out, const float* __restrict__ Q,
                                                          const __half* __restrict__ kc, const __half* __restrict__ vc,
                                                          int start_pos, int n_heads, int n_kv, float scale) {
    constexpr int HD = DPL * 32;
    extern __shared__ float smem_dyn[];
    const int head0 = blockIdx.x * GC, qi = blockIdx.y;
    const int kv_head = head0 / (n_heads / n_kv);
    const size_t qoff = ((size_t)qi * n_heads + head0) * HD;
    attend_group<DPL, GC>(out + qoff, Q + qoff, kc, vc, kv_head, n_kv, 0, start_pos + qi + 1, scale, nullptr, nullptr, smem_dyn);
}

int pick_gc(int group) { return group % 8 == 0 ? 8 : group % 4 == 0 ? 4 : group % 2 == 0 ? 2 : 1; }

constexpr int wave(int gc, int hd) { return 148 * (hd == 64 && gc <= 2 ? 3 : 2); }      // CTAs of the walk that are resident at once: those of narrow heads have 80 registers
// Slices of the keys of one query that the scratch of a captured step has room for, `groups` CTAs to a slice: at least 32 keys each, two CTAs to an SM
int wave_splits(int keys, int groups) { return std::max(1, std::min({2 * 148 / groups, (keys + 31) / 32, MAX_SPLITS})); }

// Slices of a run of `tokens` queries over `total` keys, `groups` CTAs to a query and a slice: at least 32 keys each, at most three waves of CTAs.
int rows_splits_most(int tokens, int total, int groups, int gc, int hd) { return std::max(1, std::min({3 * wave(gc, hd) / (groups * tokens), (total + 31) / 32, MAX_SPLITS})); }
// A CTA takes 1.25 us and then, for a key, 10.6 ns and 1.5 ns for each query head that shares it (of 128), 1.5 times that beside others on its SM; an SM takes its CTAs two at a time,
// three where they are narrow (more than 74 CTAs are two to an SM: those that wait for the launch before gather).  The merge takes 3.5 us and 6 us for a million of the slices' sums.
// Fitted to 784 calls (2 to 31 tokens, 4 to 48 groups, all widths, 0 to 1900 keys before).  As many slices as fill two CTAs to an SM and one more, and
// these, us: 21 tokens, 32 heads of 128 over 8, behind 30, 120, 300, 1900: 10.5, 4.9; 12.6, 7.8; 17.1, 13.3; 56.5, 50.8; 16 heads of 64, 16 behind 1900: 41.3, 37.1; the mean takes
// 0.89 of the time.  (By waves of two CTAs to an SM whatever their width, each begun at 0.7 of one: 56.9 there, and 40 heads of 128 over 8, 11 behind 1000 41.9 in two slices, 38.7
// whole.)  Eight heads of 128 to a key head stay with the former: their sums are one run (attention_walk.cuh), and longer slices would cost precision (31 queries behind 1000:
// 2.2e-7, 2.6e-7).
int rows_splits(int tokens, int total, int groups, int gc, int hd) {
    if (gc * hd > 512) return std::max(1, std::min({(2 * 148 + groups * tokens - 1) / (groups * tokens), (total + 31) / 32, MAX_SPLITS}));
    const float key = 0.0106f + 0.0015f * gc * hd / 128;
    const int at_once = wave(gc, hd) / 148;
    int best = 1;
    float least = 0.f;
    for (int n = 1, most = rows_splits_most(tokens, total, groups, gc, hd); n <= most; n++) {
        const int len = (total + n - 1) / n, used = (total + len - 1) / len, ctas = groups * tokens * used, to_an_sm = ctas > 74 ? std::max(2, (ctas + 147) / 148) : 1, left = to_an_sm % at_once;
        const float walked = (float)((to_an_sm - left) / at_once + (left > 1)) * (1.25f + 1.5f * key * len) + (left == 1 ? 1.25f + key * len : 0.f);
        const float t = used > 1 ? walked + 3.5f + 6e-6f * used * tokens * groups * gc * hd : walked;
        if (n == 1 || t < least) { least = t; best = used; }
    }
    return best;
}
// Of a single query.  As many as fit a wave of two CTAs to an SM: one slice more began a second wave (32 heads of 128 with keys of their own, 700, 2000 and 6000 keys: 8.4, 7.0;
// 13.0, 9.8; 30.2, 22.1; 24 heads over 8, 4000 keys, 13 and 12: 15.8, 12.6).  One more where three fit (64 heads of 64, 2000 and 6000 keys, four and five: 18.5, 16.2; 50.6, 41.9).
// Groups of more than half a wave would have one slice however many keys: up to three quarters of one, by what they cost, narrow ones two at least from 400 keys on (one, two and these:
// 160 groups of 128, 2000 and 6000 keys 53.9, 50.4, 41.0; 151, 136, 102; 160 of 64, 6000: 141, 96.9, 74.7; 256 of 64, 700 and 2000: 22.3, 18.4, 18.4; 64.7, 50.8, 44.5);
// beyond, memory is what bounds (240 of 128, 2000 keys, one and two: 55.3, 58.4).
int decode_splits(int keys, int groups, int gc, int hd) {
    if (keys <= 64) return 1;
    const bool narrow = wave(gc, hd) > 296;
    if (groups > 148) return groups > wave(gc, hd) * 3 / 4 ? 1 : std::max(narrow && keys >= 400 ? 2 : 1, rows_splits(1, keys, groups, gc, hd));
    return narrow ? std::min({(295 + groups) / groups, (keys + 31) / 32, MAX_SPLITS}) : wave_splits(keys, groups);
}
template <int DPL, int GC>
void launch_decode(float* out, const float* q, const __half* kc, const __half* vc, int seq_len, int n_heads, int n_kv,
                   float scale, cudaStream_t s) {
    constexpr int HD = DPL * 32;
    int groups = n_heads / GC;
    int n_splits = decode_splits(seq_len, groups, GC, HD);
    int split_len = (seq_len + n_splits - 1) / n_splits;
    n_splits = (seq_len + split_len - 1) / split_len;
    const size_t smem = ((size_t)walk_floats<DPL, GC>() + (size_t)GC * HD + 2 * GC) * sizeof(float);
    static unsigned long long configured[2] = {};      // bit per device id
    // sums apart where the groups do not fill the wave, so that the slices are longer (32 groups, 2000 keys: 1.94e-7 of error, 1.81e-7 so); elsewhere they cost 1 % and nothing calls for them
    const bool apart = 296 % groups != 0;
    auto kernel = apart ? decode_kernel<DPL, GC, true> : decode_kernel<DPL, GC, false>;
    opt_in_dynamic_smem(kernel, (int)(ATTN_MAX_DYN_SMEM), configured[apart]);
    // the slices' results: the stream's, so that calls on other streams and devices and by other threads have their own
    std::optional<StreamMemory> memory;
    if (n_splits > 1) memory.emplace((size_t)n_heads * n_splits * (HD + 2) * sizeof(float), s);
    float* scratch = memory ? static_cast<float*>(memory->p) : nullptr;
    if (!scratch) { n_splits = 1; split_len = seq_len; }          // no memory: one slice
    // Programmatic launches outside graphs too: neither kernel reads or writes before its wait, so the merge's launch hides behind the slices
    launch_k_pdl(true, kernel, dim3(groups, n_splits), dim3(AW * 32), smem, s, out, q, kc, vc, seq_len, n_heads, n_kv, scale, n_splits, split_len,
                 scratch, (const int*)nullptr);
    count_launch();
    if (n_splits > 1) {
        launch_k_pdl(true, decode_combine_kernel, dim3(n_heads), dim3(128), 0, s, out, (const float*)scratch, n_heads, HD, n_splits, seq_len, split_len, (const int*)nullptr,
                     (int8_t*)nullptr);
        count_launch();
    }
}

// A few consecutive queries (start_pos ...), each with the arithmetic of a decoded token; scratch: attention_rows_scratch_floats().
template <int DPL, int GC>
void launch_rows(float* out, const float* q, const __half* kc, const __half* vc, int tokens, int start_pos, int n_heads, int n_kv, float scale, float* scratch,
                 cudaStream_t s) {
    constexpr int HD = DPL * 32;
    const int groups = n_heads / GC, total = start_pos + tokens;
    int n_splits = rows_splits(tokens, total, groups, GC, HD);
    const int split_len = (total + n_splits - 1) / n_splits;
    n_splits = (total + split_len - 1) / split_len;
    const size_t smem = ((size_t)walk_floats<DPL, GC>() + (size_t)GC * HD + 2 * GC) * sizeof(float);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(decode_kernel<DPL, GC>, (int)(ATTN_MAX_DYN_SMEM), configured);
    NT_CHECK(n_splits <= MAX_SPLITS, "attention over a run of tokens: context beyond the slices");
    launch_k_pdl(true, decode_kernel<DPL, GC>, dim3(groups, n_splits, tokens), dim3(AW * 32), smem, s, out, q, kc, vc, start_pos + 1, n_heads, n_kv, scale, n_splits, split_len,
             scratch, (const int*)nullptr);
    count_launch();
    if (n_splits > 1) {
        launch_k_pdl(true, decode_combine_kernel, dim3(n_heads, tokens), dim3(128), 0, s, out, (const float*)scratch, n_heads, HD, n_splits, start_pos + 1, split_len,
                 (const int*)nullptr, (int8_t*)nullptr);
        count_launch();
    }
}

// Graph-replayable decode: the context length (pos + 1) is read from device memory, the launch shape is fixed
// by max_seq, partials always go through caller-owned scratch (n_heads * n_splits * (HD + 2) floats).
template <int DPL, int GC>
void launch_decode_dyn(float* out, const float* q, const __half* kc, const __half* vc, const int* pos_dev, int max_seq,
                       int n_heads, int n_kv, float scale, float* scratch, int n_splits, int8_t* xq_out, cudaStream_t s) {
    constexpr int HD = DPL * 32;
    const int groups = n_heads / GC;
    const size_t smem = ((size_t)walk_floats<DPL, GC>() + (size_t)GC * HD + 2 * GC) * sizeof(float);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(decode_kernel<DPL, GC>, (int)(ATTN_MAX_DYN_SMEM), configured);
    launch_k(decode_kernel<DPL, GC>, dim3(groups, n_splits), dim3(AW * 32), smem, s, out, q, kc, vc, 0, n_heads, n_kv, scale,
             n_splits, 0, scratch, pos_dev);
    launch_k(decode_combine_kernel, dim3(n_heads), dim3(128), 0, s, out, (const float*)scratch, n_heads, HD, n_splits, 0, 0, pos_dev, xq_out);
    count_launch(2);
}

template <int DPL, int GC>
void launch_decode_fused(float* out, const float* q, const float* k_new, const float* v_new, __half* kc, __half* vc, const int* pos_dev,
                         int max_seq, int n_heads, int n_kv, float theta, float freq_scale, float scale, float* scratch, int n_splits,
                         unsigned* tickets, int8_t* xq_out, cudaStream_t s) {
    constexpr int HD = DPL * 32;
    const int groups = n_heads / GC;
    const size_t smem = ((size_t)walk_floats<DPL, GC>() + (size_t)GC * HD + 2 * GC) * sizeof(float);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(decode_fused_kernel<DPL, GC>, (int)(ATTN_MAX_DYN_SMEM), configured);
    launch_k(decode_fused_kernel<DPL, GC>, dim3(groups, n_splits), dim3(AW * 32), smem, s, out, q, k_new, v_new, kc, vc, pos_dev, n_heads,
             n_kv, scale, theta, freq_scale, n_splits, FUSED_MIN_SPLIT, scratch, tickets, xq_out);
    count_launch();
}

// RoPE + KV write folded into the split-context decode kernel, merge as its own small launch (same slices as launch_decode_dyn):
// two launches instead of rope_kv_decode + decode + combine, without the one-launch form's serial chain or tickets.
template <int DPL, int GC>
void launch_decode_rope_dyn(float* out, const float* q, const float* k_new, const float* v_new, __half* kc, __half* vc, const int* pos_dev,
                            int max_seq, int n_heads, int n_kv, float theta, float freq_scale, float scale, float* scratch, int n_splits,
                            int8_t* xq_out, cudaStream_t s) {
    constexpr int HD = DPL * 32;
    const int groups = n_heads / GC;
    const size_t smem = ((size_t)walk_floats<DPL, GC>() + (size_t)GC * HD + 2 * GC) * sizeof(float);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(decode_fused_kernel<DPL, GC>, (int)(ATTN_MAX_DYN_SMEM), configured);
    launch_k(decode_fused_kernel<DPL, GC>, dim3(groups, n_splits), dim3(AW * 32), smem, s, out, q, k_new, v_new, kc, vc, pos_dev, n_heads,
             n_kv, scale, theta, freq_scale, n_splits, DYN_MIN_SPLIT, scratch, (unsigned*)nullptr, (int8_t*)nullptr);
    launch_k(decode_combine_kernel, dim3(n_heads), dim3(128), 0, s, out, (const float*)scratch, n_heads, HD, n_splits, 0, 0, pos_dev, xq_out);
    count_launch(2);
}

template <int DPL, int GC>
void launch_prefill(float* out, const float* Q, const __half* kc, const __half* vc, int seq_len, int start_pos, int n_heads,
                    int n_kv, float scale, cudaStream_t s) {
    const size_t smem = (size_t)walk_floats<DPL, GC>() * sizeof(float);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(prefill_kernel<DPL, GC>, (int)(ATTN_MAX_DYN_SMEM), configured);
    prefill_kernel<DPL, GC><<<dim3(n_heads / GC, seq_len), AW * 32, smem, s>>>(out, Q, kc, vc, start_pos, n_heads, n_kv, scale);
    count_launch();
}

#define NT_DISPATCH_ATTN(FN, ...)                                                         \
    do {                                                                                  \
        const int gc_ = pick_gc(n_heads / n_kv);                                          \
        const int dpl_ = hd / 32;                                                         \
        NT_CHECK(hd % 32 == 0 && (dpl_ == 2 || dpl_ == 4 || dpl_ == 8),                  \
                 "attention: head_dim must be 64, 128 or 256");                           \
        NT_CHECK(n_kv > 0 && n_heads % n_kv == 0, "attention: n_heads % n_kv_heads != 0"); \
        if (dpl_ == 4) {                                                                  \
            if (gc_ == 8) FN<4, 8>(__VA_ARGS__); else if (gc_ == 4) FN<4, 4>(__VA_ARGS__); \
            else if (gc_ == 2) FN<4, 2>(__VA_ARGS__); else FN<4, 1>(__VA_ARGS__);         \
        } else if (dpl_ == 2) {                                                           \
            if (gc_ == 8) FN<2, 8>(__VA_ARGS__); else if (gc_ == 4) FN<2, 4>(__VA_ARGS__); \
            else if (gc_ == 2) FN<2, 2>(__VA_ARGS__); else FN<2, 1>(__VA_ARGS__);         \
        } else {                                                                          \
            if (gc_ == 8) FN<8, 8>(__VA_ARGS__); else if (gc_ == 4) FN<8, 4>(__VA_ARGS__); \
            else if (gc_ == 2) FN<8, 2>(__VA_ARGS__); else FN<8, 1>(__VA_ARGS__);         \
        }                                                                                 \
    } while (0)

}  // namespace

void attention_decode(float* out, const float* q, const void* kc, const void* vc, int seq_len, int n_heads, int n_kv,
                      int hd, int max_seq, float scale, cudaStream_t s) {
    if (seq_len <= 0 || n_heads <= 0) return;
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
    NT_DISPATCH_ATTN(launch_decode, out, q, k, v, seq_len, n_heads, n_kv, scale, s);
}

size_t attention_rows_scratch_floats(int tokens, int max_seq, int n_heads, int n_kv, int hd) {
    const int gc = pick_gc(n_heads / n_kv);
    size_t most = 0;                     // fewer tokens are cut into more slices
    for (int t = 1; t <= tokens; t++) most = std::max(most, (size_t)t * n_heads * rows_splits_most(t, max_seq, n_heads / gc, gc, hd) * (hd + 2));
    return most;
}
void attention_rows_f16(float* out, const float* q, const void* kc, const void* vc, int tokens, int start_pos, int n_heads, int n_kv, int hd, float scale,
                        float* scratch, cudaStream_t s) {
    if (tokens <= 0 || n_heads <= 0) return;
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
    NT_DISPATCH_ATTN(launch_rows, out, q, k, v, tokens, start_pos, n_heads, n_kv, scale, scratch, s);
}

int attention_decode_dyn_splits(int max_seq, int n_heads, int n_kv) { return wave_splits(max_seq, n_heads / pick_gc(n_heads / n_kv)); }
size_t attention_decode_dyn_scratch_floats(int max_seq, int n_heads, int n_kv, int hd) {
    return (size_t)n_heads * attention_decode_dyn_splits(max_seq, n_heads, n_kv) * (hd + 2);
}
void attention_decode_dyn(float* out, const float* q, const void* kc, const void* vc, const int* pos_dev, int max_seq,
                          int n_heads, int n_kv, int hd, float scale, float* scratch, void* xq_out, cudaStream_t s) {
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
    const int n_splits = attention_decode_dyn_splits(max_seq, n_heads, n_kv);
    if (xq_out) NT_CHECK((n_heads * hd) % 128 == 0, "attention_decode_dyn: n_heads * head_dim must be a multiple of 128 for the fused quantiser");
    NT_DISPATCH_ATTN(launch_decode_dyn, out, q, k, v, pos_dev, max_seq, n_heads, n_kv, scale, scratch, n_splits, static_cast<int8_t*>(xq_out), s);
}

int attention_decode_fused_tickets(int n_heads, int n_kv) { return n_heads / pick_gc(n_heads / n_kv); }
void attention_decode_fused(float* out, const float* q, const float* k, const float* v, void* kc, void* vc, const int* pos_dev,
                            int max_seq, int n_heads, int n_kv, int hd, float theta, float freq_scale, float scale, float* scratch,
                            unsigned* tickets, void* xq_out, cudaStream_t s) {
    __half* kh = static_cast<__half*>(kc);
    __half* vh = static_cast<__half*>(vc);
    const int n_splits = attention_decode_dyn_splits(max_seq, n_heads, n_kv);
    if (xq_out) NT_CHECK((n_heads * hd) % 128 == 0, "attention_decode_fused: n_heads * head_dim must be a multiple of 128 for the fused quantiser");
    NT_DISPATCH_ATTN(launch_decode_fused, out, q, k, v, kh, vh, pos_dev, max_seq, n_heads, n_kv, theta, freq_scale, scale, scratch, n_splits,
                     tickets, static_cast<int8_t*>(xq_out), s);
}

void attention_decode_rope_dyn(float* out, const float* q, const float* k, const float* v, void* kc, void* vc, const int* pos_dev,
                               int max_seq, int n_heads, int n_kv, int hd, float theta, float freq_scale, float scale, float* scratch,
                               void* xq_out, cudaStream_t s) {
    __half* kh = static_cast<__half*>(kc);
    __half* vh = static_cast<__half*>(vc);
    const int n_splits = attention_decode_dyn_splits(max_seq, n_heads, n_kv);
    if (xq_out) NT_CHECK((n_heads * hd) % 128 == 0, "attention_decode_rope_dyn: n_heads * head_dim must be a multiple of 128 for the fused quantiser");
    NT_DISPATCH_ATTN(launch_decode_rope_dyn, out, q, k, v, kh, vh, pos_dev, max_seq, n_heads, n_kv, theta, freq_scale, scale, scratch, n_splits,
                     static_cast<int8_t*>(xq_out), s);
}

// Whether a prompt is better served by the tiles of 128 queries x 128 keys on tcgen05 (one CTA to an SM and two of these tiles, which walk all keys in series, however few
// of their rows are live) than by those of 64 x 64 on mma.sync.  Beyond a wave of the smaller tiles always (500 tokens, 24 heads of 128: 21.5 us, 31.8 on mma.sync; 1000
// behind 1023, 32 heads: 57, 174).  Within one, each takes a start and its steps over the keys of the last query, heads of 128 (64): 8.4 us and 2.82 (5.8 and 2.1) for
// 128 keys here, 5.6 us and 1.9 (4.5 and 1.22) for 64 keys there, and 0.7 (0.3) more here each time the queries' tiles double.  Measured (here, there): 17 tokens
// behind 0, 300, 1000: 10.9, 16.8, 31.0; 8.4, 14.5, 36.1 (heads of 64: 7.8, 12.3, 22.9; 6.3, 10.5, 24.7); 200 behind 0, 300: 14.6, 21.9; 12.5, 22.7.  Of 720 pairs (17 to 1000 tokens, 4 to 64 heads,
// 0 to 4000 keys before, both widths) none takes a form that is more than 3 % slower, but 12 of heads of 64, by up to 6 %, on mma.sync.
bool attention_prefill_tc_pays(int seq_len, int start_pos, int n_heads, int hd) {
    if ((long long)((seq_len + 63) / 64) * n_heads > 148) return true;
    const int keys = start_pos + seq_len;
    const float s64 = (float)((keys + 63) / 64), s128 = (float)((keys + 127) / 128), doubled = log2f((float)((seq_len + 127) / 128));
    return hd == 128 ? 1.9f * s64 - 2.82f * s128 - 0.7f * doubled > 2.75f : 1.22f * s64 - 2.1f * s128 - 0.3f * doubled > 1.25f;
}
// How many slices the keys are cut into.  Either form walks a CTA's keys in series, and where the queries give fewer CTAs than there are SMs, the rest idle: slices, at the
// price of writing their sums and reading them again.  Times as measured (us): the tcgen05 form 8.0 and 1.5 for 64 keys (heads of 64: 4.5 and 1.2), the whole one on
// mma.sync 5.5 and 2.1 (4.2 and 1.3); slices with their merge 6.0 and 2.3 (1.4) for 64 keys of one, 1.7 (1.5) times that where two CTAs share an SM, and the sums at
// 0.35 us a megabyte; a slice more costs 0.2.  Whole, in slices: heads of 128, 8 of them, 40 tokens behind 965: 31.2, 13.2; 64, 17 behind 1000: 32.1, 22.8; 2, 1500 behind
// 1500: 78.3, 39.3; 8, 518 behind 5: 24.2, 21.4; heads of 64, 16 of them, 60 behind 700: 18.8, 10.5.  Not cut: 32 heads of 128, 256 behind 0: 14.4, 18.8 in two;
// 64 heads, 128 behind 1000: 37.0, 42.5.  Cut only where 2.2 us are gained by that account, which is out by as much where tiles are few (16 heads, 224 behind 0: 12.6, 14.6 in
// two): of 768 calls with less than a wave of CTAs none is then slower, and the mean takes 0.71 of the time.
// Between programmatic launches the plain one costs 3 to 4 us more: 60 tokens behind 900, 32 heads of 128, two layers of 4096: 443 us whole, 426 in slices.
int attention_prefill_slices_for(int form, int seq_len, int start_pos, int n_heads, int hd, int max_seq, bool in_chain) {
    const long long ctas = (long long)((seq_len + 63) / 64) * n_heads, tiles = ((long long)start_pos + seq_len + 63) / 64;
    if (form == PREFILL_QUERIES || start_pos < 0 || (long long)start_pos + seq_len > max_seq || ctas > 148 || tiles < 4) return 1;
    const bool wide = hd == 128;
    const float whole = form == PREFILL_TC ? (wide ? 8.0f + 1.5f * tiles : 4.5f + 1.2f * tiles) : (wide ? 5.5f + 2.1f * tiles : 4.2f + 1.3f * tiles);
    const float written = 0.35e-6f * 4 * seq_len * n_heads * hd + 0.2f;       // a slice's sums, there and back
    int best = 1;
    float least = whole - (in_chain ? 5.0f : 2.2f);
    for (int n = 2; n <= 16 && n <= tiles; n++) {
        const long long all = ctas * n, steps = (tiles + n - 1) / n * ((all + 295) / 296);
        const float t = 6.0f + (wide ? 2.3f : 1.4f) * steps * (all <= 148 ? 1.0f : wide ? 1.7f : 1.5f) + n * written;
        if (t < least) { least = t; best = n; }
    }
    return best;
}
// prompt-sized chunks: tiled tensor-core kernels
int attention_prefill_form(const float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads, int n_kv, int hd, int max_seq, bool in_chain) {
    if (!attention_prefill_mma_supported(seq_len, n_heads, n_kv, hd)) return PREFILL_QUERIES;
    return attention_prefill_tc_takes(out, Q, kc, vc, seq_len, start_pos, n_heads, n_kv, hd, max_seq) && (in_chain || attention_prefill_tc_pays(seq_len, start_pos, n_heads, hd))
               ? PREFILL_TC : PREFILL_MMA;
}
void attention_prefill(float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads,
                       int n_kv, int hd, int max_seq, float scale, cudaStream_t s, bool in_chain) {
    if (seq_len <= 0 || n_heads <= 0) return;
    const int form = attention_prefill_form(out, Q, kc, vc, seq_len, start_pos, n_heads, n_kv, hd, max_seq, in_chain);
    if (form != PREFILL_QUERIES) {
        const int slices = attention_prefill_slices_for(form, seq_len, start_pos, n_heads, hd, max_seq, in_chain);
        if (slices > 1 && attention_prefill_slices(out, Q, kc, vc, seq_len, start_pos, n_heads, n_kv, hd, max_seq, scale, slices, s)) return;
        if (form == PREFILL_TC && attention_prefill_tc(out, Q, kc, vc, seq_len, start_pos, n_heads, n_kv, hd, scale, s)) return;
        attention_prefill_mma(out, Q, kc, vc, seq_len, start_pos, n_heads, n_kv, hd, max_seq, scale, s);
        return;
    }
    const __half* k = static_cast<const __half*>(kc);
    const __half* v = static_cast<const __half*>(vc);
    NT_DISPATCH_ATTN(launch_prefill, out, Q, k, v, seq_len, start_pos, n_heads, n_kv, scale, s);
}

}}  // namespace nt::b200
