// attention_row.cuh — a row of prompt attention by itself: what both forms on the tensor cores do for rows that these left infinite or NaN.
#pragma once
#include <cuda_fp16.h>

namespace nt { namespace b200 { namespace {

// A row by itself, HC of its channels, by a warp: keys 0 .. pos and no others, 32 at a time, a key to a lane and then HC / 32 channels to each.  For a row whose sums the
// products left infinite or NaN: the weight of a key that the row does not see is zero, and zero times an infinite or NaN value, of a later token in the row's last
// steps, is NaN.  Values that the row does see reach it here as well.
template <int HD, int HC, class Attn>
__device__ __noinline__ void row_alone(const Attn& p, int row, int head, int channel, int lane) {
    constexpr int C = HC / 32;
    const size_t pitch = (size_t)p.n_kv * HD, at = ((size_t)row * p.n_heads + head) * HD;
    const int pos = p.start_pos + row;
    const size_t kvh = (size_t)(head / (p.n_heads / p.n_kv));
    const __half* k = p.kc + kvh * HD;
    const __half* v = p.vc + kvh * HD + channel + lane * C;
    float m = -INFINITY, l = 0.f, o[C] = {};
#pragma unroll 1
    for (int k0 = 0; k0 <= pos; k0 += 32) {
        float s = 0.f;
        const __half* kr = k + (size_t)min(k0 + lane, pos) * pitch;
#pragma unroll 4
        for (int d = 0; d < HD; d += 2) {
            const float2 x = __half22float2(*reinterpret_cast<const __half2*>(kr + d)), q = *reinterpret_cast<const float2*>(p.Q + at + d);
            s = fmaf(q.x, x.x, fmaf(q.y, x.y, s));
        }
        s = k0 + lane <= pos ? s * p.scale * 1.4426950408889634f : -INFINITY;
        float mx = fmaxf(m, s);
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, i));
        const float base = mx == -INFINITY ? 0.f : mx, alpha = exp2f(m - base), w = exp2f(s - base);
        m = mx;
        float sum = w;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, i);
        l = fmaf(l, alpha, sum);
#pragma unroll
        for (int i = 0; i < C; i++) o[i] *= alpha;
        for (int j = 0; j < min(32, pos + 1 - k0); j++) {
            const float wj = __shfl_sync(0xFFFFFFFFu, w, j);
#pragma unroll
            for (int i = 0; i < C; i++) o[i] = fmaf(wj, __half2float(v[(size_t)(k0 + j) * pitch + i]), o[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < C; i++) p.out[at + channel + lane * C + i] = o[i] / l;
}

}}}  // namespace nt::b200::(anonymous)
