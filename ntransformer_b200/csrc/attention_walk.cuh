// attention_walk.cuh — one CTA's walk over a slice of the F16 cache for the query heads that share a key head: the same arithmetic, key by key and
// merge by merge, in the decode kernels (attention.cu) and in the persistent decode-step kernel (engine/decode_megakernel.cu).
//
// Bound by latency: a slice has few keys to a warp.  Each warp takes batches of KU consecutive keys with a running maximum of its own, so nothing waits for
// another warp before the end, and the next batch's keys are on their way while the weights are formed, its values while the next scores are
// (a form that walked the slice three times, scores, softmax, values, with a barrier and a fetch in front of each: 64 heads, 8 key heads, 4000 keys
// 12.6 + 5 us for the slices and their merge, 21 us a call; this one 14.5).
#pragma once
#include <cuda_fp16.h>
#include <cfloat>
#include <cstdint>

namespace nt { namespace b200 {
namespace {

constexpr int WALK_WARPS = 8;            // warps of a CTA that walk
constexpr int KU = 8;                    // cache rows a warp keeps in flight
constexpr int P_LD = KU + 1;             // per warp: KU weights and the rescaling of what is summed so far, for each head

template <int N> struct HalfVec;         // N halfs loaded as one vector
template <> struct HalfVec<2> { using T = uint32_t; };
template <> struct HalfVec<4> { using T = uint2; };
template <> struct HalfVec<8> { using T = uint4; };

// Reduce GC per-lane partial sums across the warp. On return lane L holds (in v[0]) the full sum of
// value index (L / (32 / GC)) ... valid in every lane of that group.
template <int GC>
__device__ __forceinline__ float transpose_reduce(float (&v)[GC], int lane) {
    // exchange phase: halve the number of live values per step
#pragma unroll
    for (int n = GC, off = 16; n > 1; n >>= 1, off >>= 1) {
        const bool upper = lane & off;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            float send = upper ? v[i] : v[i + n / 2];
            float keep = upper ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, off);
        }
    }
    // plain butterfly over the remaining lanes of the group
    float r = v[0];
#pragma unroll
    for (int off = 16 / GC; off > 0; off >>= 1) r += __shfl_xor_sync(0xFFFFFFFFu, r, off);
    return r;
}

// Shared memory of a walk, in floats: weights [warp][KU + 1][GC], sums [warp][GC][HD], (maximum, sum) [warp][GC][2].
template <int DPL, int GC> __host__ __device__ constexpr int walk_floats() { return WALK_WARPS * GC * P_LD + WALK_WARPS * GC * DPL * 32 + 2 * WALK_WARPS * GC; }

// Warp `warp` of WALK_WARPS, keys [k_begin, k_end).  kbase, vbase: this lane's DPL channels of cache row 0.  load_q(qr) gives the lane's channels of the
// queries (after the first rows are under way).  OWN: row `own` is not read from the cache, own_key(f) and own_value(f) give it.
// APART: eight keys' sums apart, see below.
template <int DPL, int GC, bool OWN, bool APART, class LoadQ, class OwnKey, class OwnValue>
__device__ __forceinline__ void walk_slice(const __half* kbase, const __half* vbase, size_t row_stride, int k_begin, int k_end, int own, float scale, float* smem,
                                           int warp, int lane, LoadQ load_q, OwnKey own_key, OwnValue own_value) {
    constexpr int HD = DPL * 32, LG = 32 / GC;           // lanes that hold a head's score
    using Raw = typename HalfVec<DPL>::T;
    // Eight keys' sums by themselves before they join the run's, whose length then costs less: 1900 keys in two slices 2.6e-7 of error in one run, 1.8e-7 so.  Not where
    // the registers do not hold both (64 heads over 8: 4000 keys 12.3 us, 13.6 so; 27 queries behind 1900 85, 102).
    constexpr bool BLOCKED = APART && DPL * GC <= 16;
    // Two chains of them, even and odd keys; one where two heads of 256 leave no registers for both (8 heads over 4, 15 queries behind 1500: 35.0 us in one run, 45.5 with two
    // chains, 38.9 with one; 16 over 8, 6000 keys: 13.4, 14.8, 13.7)
    constexpr int CHAINS = DPL == 8 && GC == 2 ? 1 : 2;
    float* pw = smem + (size_t)warp * GC * P_LD;
    float* red = smem + (size_t)WALK_WARPS * GC * P_LD;
    float* ml = red + (size_t)WALK_WARPS * GC * HD;

    Raw kr[KU] = {}, vr[KU] = {};
    auto fetch = [&](const __half* base, Raw (&r)[KU], int k0) {     // rows behind the slice are its last one: loaded, not used
#pragma unroll
        for (int u = 0; u < KU; u++) {
            const int row = k0 + u < k_end - 1 ? k0 + u : k_end - 1;
            if (!OWN || row != own) r[u] = __ldg(reinterpret_cast<const Raw*>(base + (size_t)row * row_stride));
        }
    };
    auto to_float = [](const Raw& raw, float (&f)[DPL]) {
        const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
        for (int i = 0; i < DPL / 2; i++) { const float2 t = __half22float2(h2[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
    };
    int k0 = k_begin + warp * KU;
    if (k0 < k_end) { fetch(kbase, kr, k0); fetch(vbase, vr, k0); }

    float qr[GC][DPL];
    load_q(qr);
    float acc[GC][DPL];
#pragma unroll
    for (int g = 0; g < GC; g++)
#pragma unroll
        for (int i = 0; i < DPL; i++) acc[g][i] = 0.f;
    float mx = -FLT_MAX, sum = 0.f;                      // of head lane / LG
    for (; k0 < k_end; k0 += WALK_WARPS * KU) {
        float s[KU];
#pragma unroll
        for (int u = 0; u < KU; u++) {
            float kf[DPL];
            to_float(kr[u], kf);
            if (OWN && k0 + u == own) own_key(kf);              // warp-uniform
            float part[GC];
#pragma unroll
            for (int g = 0; g < GC; g++) {
                float a = 0.f;
#pragma unroll
                for (int i = 0; i < DPL; i++) a = fmaf(qr[g][i], kf[i], a);
                part[g] = a;
            }
            const float tot = transpose_reduce<GC>(part, lane) * scale;
            s[u] = k0 + u < k_end ? tot : -FLT_MAX;
        }
        if (k0 + WALK_WARPS * KU < k_end) fetch(kbase, kr, k0 + WALK_WARPS * KU);
        float m2 = mx;
#pragma unroll
        for (int u = 0; u < KU; u++) m2 = fmaxf(m2, s[u]);
        const float corr = expf(mx - m2);                // the first batch: 0, or 1 where no score lies above -FLT_MAX (then the sums are 0)
        mx = m2;
        if constexpr (BLOCKED) {
#pragma unroll
            for (int u = 0; u < KU; u++) s[u] = k0 + u < k_end ? expf(s[u] - m2) : 0.f;
            sum = fmaf(sum, corr, ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7])));
        } else {
            sum *= corr;
#pragma unroll
            for (int u = 0; u < KU; u++) {
                s[u] = k0 + u < k_end ? expf(s[u] - m2) : 0.f;
                sum += s[u];
            }
        }
        __syncwarp();                                    // the weights of the batch before have been read
        if ((lane & (LG - 1)) == 0) {
#pragma unroll
            for (int u = 0; u < KU; u++) pw[u * GC + lane / LG] = s[u];
            pw[KU * GC + lane / LG] = corr;
        }
        __syncwarp();
        if constexpr (BLOCKED) {
            float part[CHAINS][GC][DPL] = {};
#pragma unroll
            for (int u = 0; u < KU; u++) {
                if (k0 + u >= k_end) break;
                float vf[DPL];
                to_float(vr[u], vf);
                if (OWN && k0 + u == own) own_value(vf);
#pragma unroll
                for (int g = 0; g < GC; g++) {
                    const float w = pw[u * GC + g];
#pragma unroll
                    for (int i = 0; i < DPL; i++) part[u % CHAINS][g][i] = fmaf(w, vf[i], part[u % CHAINS][g][i]);
                }
            }
#pragma unroll
            for (int g = 0; g < GC; g++) {
                const float c = pw[KU * GC + g];
#pragma unroll
                for (int i = 0; i < DPL; i++) acc[g][i] = fmaf(acc[g][i], c, CHAINS == 2 ? part[0][g][i] + part[CHAINS - 1][g][i] : part[0][g][i]);
            }
        } else {
#pragma unroll
            for (int g = 0; g < GC; g++) {
                const float c = pw[KU * GC + g];
#pragma unroll
                for (int i = 0; i < DPL; i++) acc[g][i] *= c;
            }
#pragma unroll
            for (int u = 0; u < KU; u++) {
                if (k0 + u >= k_end) break;
                float vf[DPL];
                to_float(vr[u], vf);
                if (OWN && k0 + u == own) own_value(vf);
#pragma unroll
                for (int g = 0; g < GC; g++) {
                    const float w = pw[u * GC + g];
#pragma unroll
                    for (int i = 0; i < DPL; i++) acc[g][i] = fmaf(w, vf[i], acc[g][i]);
                }
            }
        }
        if (k0 + WALK_WARPS * KU < k_end) fetch(vbase, vr, k0 + WALK_WARPS * KU);
    }
#pragma unroll
    for (int g = 0; g < GC; g++)
#pragma unroll
        for (int i = 0; i < DPL; i++) red[((size_t)warp * GC + g) * HD + lane * DPL + i] = acc[g][i];
    if ((lane & (LG - 1)) == 0) { ml[(warp * GC + lane / LG) * 2] = mx; ml[(warp * GC + lane / LG) * 2 + 1] = sum; }
}

// After a barrier: channel idx = g * HD + d of the slice, unnormalised (t), with its head's maximum m and sum l.
template <int DPL, int GC>
__device__ __forceinline__ void walk_merge(const float* smem, int idx, float& m, float& l, float& t) {
    constexpr int HD = DPL * 32;
    const float* red = smem + (size_t)WALK_WARPS * GC * P_LD;
    const float* ml = red + (size_t)WALK_WARPS * GC * HD;
    const int g = idx / HD;
    m = -FLT_MAX; l = 0.f; t = 0.f;
#pragma unroll
    for (int w = 0; w < WALK_WARPS; w++) m = fmaxf(m, ml[(w * GC + g) * 2]);
#pragma unroll
    for (int w = 0; w < WALK_WARPS; w++) {               // a warp without keys has sums of 0
        const float f = expf(ml[(w * GC + g) * 2] - m);
        l = fmaf(ml[(w * GC + g) * 2 + 1], f, l);
        t = fmaf(red[(size_t)w * GC * HD + idx], f, t);
    }
}

}  // namespace
}}  // namespace nt::b200
