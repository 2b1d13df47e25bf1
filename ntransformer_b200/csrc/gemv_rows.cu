// gemv_rows.cu — a few tokens (the engine: to 8, Q8_0 and Q4_0 to 31) times matrices in GGUF blocks: Y[t, n] = sum_k W[n, k] X[t, k], every weight read once for 8 tokens.
//
// The reference runs its GEMV once for every prompt token (src/model/attention.cpp:144-162, ffn.cpp:96-133), and so did the engine below the length
// where the tensor-core GEMM of prompts pays: 21 tokens cost 21 decode steps.  Here the arithmetic stays the decode step's — exact s32 products of the
// weights' codes with 24-bit activations (gemv_mma_device.cuh), F32 sums — so a token's products here do not depend on how many share the
// call (K-quants go to prefill_blocks.cu from 9 tokens on: other sums, with no larger error, which do not depend on it either):
//   * one launch quantises all tokens (optionally RMSNorm) into the order in which mma.sync's B operand wants them: 8 tokens fill the operand's columns,
//     (q1, q2) of four tokens in one product, q3 of eight in another;
//   * a CTA takes 32 rows x 8 tokens.  A producer warp streams stages of 8 super-blocks of the rows and of the tokens; 16 warps share them, a
//     super-block of 16 rows each.  Bound by the instruction issue of the per-block scales (about 450 instructions for 16 rows x 256 weights x 8 tokens) where the
//     ring has two stages (Q4_K, Q4_0, Q5_K); a stage of Q6_K, of Q4_K mixed with it and of Q8_0 leaves no room for a second, so that copies and products take turns.
#include "kernels_internal.h"
#include "ring.cuh"
#include "gemv_mma_device.cuh"
#include <cuda_fp16.h>

namespace nt { namespace b200 {

namespace {

constexpr int RKW = 8, RTILES = 2, RGROUP = RTILES * MROWS;      // super-blocks of a stage, row tiles, rows of a CTA
constexpr int RWARPS = RKW * RTILES;
constexpr int XB_DIGITS = 4 * 3 * 512, XB = XB_DIGITS + 512;     // bytes of 8 tokens' super-block: digits, scales [token][8], sums [token][8]
constexpr int R_STAGES = 2;                                      // what 227 KB hold at most

struct RowsMat { const uint8_t* W; float* y; int out, groups, fmt; long long pitch; };
struct RowsParams {
    RowsMat mat[3];
    int n_mat, NB, passes, tokens, total_units, n_seg, epilogue, stages, slot;
    const uint8_t* xr;         // [pass][super-block][XB]
    unsigned* status;          // wait_status.cuh
};

// One block: the token blockIdx.x (zeros beyond the last).  x: F32 rows of K, norm_w: RMSNorm's gains or null.
__global__ void __launch_bounds__(256) quantize_rows_kernel(uint8_t* __restrict__ xr, const float* __restrict__ xin, const float* __restrict__ norm_w, float eps,
                                                            int tokens, int K) {
    __shared__ float red[8];
    const int tok = blockIdx.x, pass = tok >> 3, tk = tok & 7, NB = K / 256;
    const bool live = tok < tokens;
    const float* x = xin + (size_t)min(tok, tokens - 1) * K;
    pdl_launch_dependents();
    pdl_wait();
    float rms = 1.f;
    if (norm_w && live) {
        float ss = 0.f;
        for (int i = threadIdx.x * 4; i < K; i += 1024) { const float4 v = *reinterpret_cast<const float4*>(x + i); ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) t += red[i];
        rms = rsqrtf(t / K + eps);
    }
    for (int t8 = threadIdx.x; t8 < K / 8; t8 += 256) {           // whole warps: K / 8 is a multiple of 32
        float v[8];
        const float4 a = *reinterpret_cast<const float4*>(x + 8 * t8), b = *reinterpret_cast<const float4*>(x + 8 * t8 + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        if (norm_w)
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = __fmul_rn(v[i], __ldg(norm_w + 8 * t8 + i));
        float amax = 0.f, s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) { amax = fmaxf(amax, fabsf(v[i])); s = __fadd_rn(s, v[i]); }
        amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
        s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, 1));
        s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, 2));
        const BlockScale scale(amax, BlockScale::TOP3);
        const int e = 8 * t8, sub = (e >> 5) & 7, seg = (e >> 4) & 1, t = (e >> 2) & 3, odd = sub & 1;
        uint8_t* blk = xr + ((size_t)pass * NB + (e >> 8)) * XB;
        uint8_t* pair = blk + (sub >> 1) * 1536;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int T[4];
            scale.integers<false>(v + 4 * h, T);
            uint32_t q1, q2, q3;
            digits4(T, q1, q2, q3);
            const int c = 2 * (tk & 3), w12 = ((tk >> 2) * 2 + seg) * 4, u12 = odd ? 1024 : 0;
            *reinterpret_cast<uint32_t*>(pair + u12 + (c * 4 + t + h) * 16 + w12) = q1;
            *reinterpret_cast<uint32_t*>(pair + u12 + ((c + 1) * 4 + t + h) * 16 + w12) = q2;
            *reinterpret_cast<uint32_t*>(pair + 512 + (tk * 4 + t + h) * 16 + (odd * 2 + seg) * 4) = q3;
        }
        if ((t8 & 3) == 0) {
            float* f = reinterpret_cast<float*>(blk + XB_DIGITS);
            f[tk * 8 + sub] = live ? __fmul_rn(BlockScale::of(amax, s, BlockScale::TOP3), rms) : 0.f;
            f[64 + tk * 8 + sub] = live ? __fmul_rn(s, rms) : 0.f;
        }
    }
}

// B words of one sub-block: columns (q1, q2) of tokens 0-3 and 4-7, q3 of tokens 0-7; each k 0-15 and 16-31.
struct BWords { uint32_t a[2][2], b[2]; };
__device__ __forceinline__ void load_pair(BWords& even, BWords& odd, const uint8_t* xb, int pair, int lane) {
    const uint4 u0 = lds128(xb + pair * 1536 + lane * 16), u1 = lds128(xb + pair * 1536 + 512 + lane * 16), u2 = lds128(xb + pair * 1536 + 1024 + lane * 16);
    even.a[0][0] = u0.x; even.a[0][1] = u0.y; even.a[1][0] = u0.z; even.a[1][1] = u0.w; even.b[0] = u1.x; even.b[1] = u1.y;
    odd.a[0][0] = u2.x; odd.a[0][1] = u2.y; odd.a[1][0] = u2.z; odd.a[1][1] = u2.w; odd.b[0] = u1.z; odd.b[1] = u1.w;
}
__device__ __forceinline__ void mma16_ss0(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
// Sums of one block of elements into the accumulators: s12[j] (tokens 4 j + t) and s3 (tokens 2 t, 2 t + 1), rows g (scale sc[0]) and g + 8 (sc[1]).
__device__ __forceinline__ void take(const int (&s12)[2][4], const int (&s3)[4], const float (&sc)[2], const float (&x12)[2], const float (&x3)[2], float (&a12)[2][2], float (&a3)[2][2]) {
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            a12[j][r] = fmaf(sum_of(s12[j][2 * r], s12[j][2 * r + 1]) * x12[j], sc[r], a12[j][r]);
            a3[j][r] = fmaf((float)s3[2 * r + j] * x3[j], sc[r], a3[j][r]);
        }
}

// One super-block x 16 rows x 8 tokens.  acc12 / acc3 as in take(); mins[j][r]: what offsets subtract for token 4 j + t.
template <int FMT>
__device__ __forceinline__ void rows_block(const uint8_t* sb, int mis, const uint8_t* xb, int lane, float (&acc12)[2][2], float (&acc3)[2][2], float (&mins)[2][2]) {
    constexpr int PITCH = stage_pitch(FMT, RKW);
    const int g = lane >> 2, t = lane & 3;
    const float* xs = reinterpret_cast<const float*>(xb + XB_DIGITS);
    float a12[2][2] = {}, a3[2][2] = {}, d[2] = {1.f, 1.f};
    const uint32_t ad = smem_u32(sb) + (uint32_t)((lane & 15) * PITCH + (lane >> 4) * 16);
    uint32_t sc[2][2], qh[4];
    const uint8_t *r0 = sb + g * PITCH + mis, *p0 = r0;
    uint32_t sel = 0x3210u;
    if (FMT <= 1) {
        if (FMT == 1) ldsm4(qh, ad + 16);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint4 h = lds128(sb + (g + 8 * r) * PITCH);
            sc[r][0] = h.y & 0x3F3F3F3Fu;
            sc[r][1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
            const uint32_t m[2] = {h.z & 0x3F3F3F3Fu, ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u)};
            float mf[8];
#pragma unroll
            for (int i = 0; i < 8; i++) mf[i] = magic_byte(m[i >> 2], 0x7440u + (i & 3));
            d[r] = half_bits(h.x & 0xFFFFu);
            const float dm = half_bits(h.x >> 16);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 s0 = *reinterpret_cast<const float4*>(xs + 64 + (4 * j + t) * 8), s1 = *reinterpret_cast<const float4*>(xs + 64 + (4 * j + t) * 8 + 4);
                float v = mf[0] * s0.x;
                v = fmaf(mf[1], s0.y, v); v = fmaf(mf[2], s0.z, v); v = fmaf(mf[3], s0.w, v);
                v = fmaf(mf[4], s1.x, v); v = fmaf(mf[5], s1.y, v); v = fmaf(mf[6], s1.z, v); v = fmaf(mf[7], s1.w, v);
                mins[j][r] = fmaf(dm, v, mins[j][r]);
            }
        }
    } else if (FMT == 2) {
        const uint32_t off = smem_u32(r0) & 2u;
        sel = off ? 0x5432u : 0x3210u;
        p0 = r0 - off;
#pragma unroll
        for (int r = 0; r < 2; r++) d[r] = half_bits(*reinterpret_cast<const uint16_t*>(r0 + r * 8 * PITCH + 208));
    }
    auto word = [&](const uint8_t* p) { return __byte_perm(*reinterpret_cast<const uint32_t*>(p), *reinterpret_cast<const uint32_t*>(p + 4), sel); };
#pragma unroll
    for (int c = 0; c < 4; c++) {                                  // sub-blocks 2 c, 2 c + 1
        BWords bw[2];
        load_pair(bw[0], bw[1], xb, c, lane);
        float x12[2][2], x3[2][2];                                 // [sub-block of the pair][token]
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float2 u = *reinterpret_cast<const float2*>(xs + (4 * j + t) * 8 + 2 * c), v = *reinterpret_cast<const float2*>(xs + (2 * t + j) * 8 + 2 * c);
            x12[0][j] = u.x; x12[1][j] = u.y; x3[0][j] = v.x; x3[1][j] = v.y;
        }
        if (FMT != 2) {
            uint32_t A[2][4];                                      // [sub-block][rows g, g + 8 of k 0-15, of k 16-31]
            float scf[2][2];
            if (FMT <= 1) {
                uint32_t q[4];
                ldsm4(q, ad + (FMT == 0 ? 16 : 48) + 32 * c);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    A[0][i] = q[i] & 0x0F0F0F0Fu;
                    A[1][i] = (q[i] >> 4) & 0x0F0F0F0Fu;
                    if (FMT == 1) {
                        A[0][i] |= (c < 2 ? qh[i] << (4 - 2 * c) : qh[i] >> (2 * c - 4)) & 0x10101010u;
                        A[1][i] |= (c < 2 ? qh[i] << (3 - 2 * c) : qh[i] >> (2 * c - 3)) & 0x10101010u;
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int k = 0; k < 2; k++) scf[k][r] = magic_byte(sc[r][c >> 1], 0x7440u + 2 * (c & 1) + k);
            } else {
                constexpr int B = FMT == 3 ? 34 : 18;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint8_t* p = sb + (g + 8 * r) * PITCH + 2 * B * c;
                    auto first = [&](const uint8_t* a) { return __byte_perm(*reinterpret_cast<const uint32_t*>(a), *reinterpret_cast<const uint32_t*>(a + 4), 0x5432u); };
                    auto second = [&](const uint8_t* a) { return *reinterpret_cast<const uint32_t*>(a + B + 2); };
                    if (FMT == 3) {
                        A[0][r] = first(p + 4 * t); A[0][2 + r] = first(p + 16 + 4 * t);
                        A[1][r] = second(p + 4 * t); A[1][2 + r] = second(p + 16 + 4 * t);
                    } else {
                        const uint32_t f = first(p + 4 * t), n = second(p + 4 * t);
                        A[0][r] = ((f << 4) & 0xF0F0F0F0u) ^ 0x80808080u; A[0][2 + r] = (f & 0xF0F0F0F0u) ^ 0x80808080u;       // 16 (q - 8) as s8
                        A[1][r] = ((n << 4) & 0xF0F0F0F0u) ^ 0x80808080u; A[1][2 + r] = (n & 0xF0F0F0F0u) ^ 0x80808080u;
                    }
                    scf[0][r] = half_bits(*reinterpret_cast<const uint16_t*>(p));
                    scf[1][r] = half_bits(*reinterpret_cast<const uint16_t*>(p + B));
                }
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                int s12[2][4], s3[4];
                if (FMT <= 1) {
                    mma_us0(s12[0], A[k][0], A[k][1], A[k][2], A[k][3], bw[k].a[0][0], bw[k].a[0][1]);
                    mma_us0(s12[1], A[k][0], A[k][1], A[k][2], A[k][3], bw[k].a[1][0], bw[k].a[1][1]);
                    mma_us0(s3, A[k][0], A[k][1], A[k][2], A[k][3], bw[k].b[0], bw[k].b[1]);
                } else {
                    mma_ss0(s12[0], A[k][0], A[k][1], A[k][2], A[k][3], bw[k].a[0][0], bw[k].a[0][1]);
                    mma_ss0(s12[1], A[k][0], A[k][1], A[k][2], A[k][3], bw[k].a[1][0], bw[k].a[1][1]);
                    mma_ss0(s3, A[k][0], A[k][1], A[k][2], A[k][3], bw[k].b[0], bw[k].b[1]);
                }
                take(s12, s3, scf[k], x12[k], x3[k], a12, a3);
            }
        } else {
            // Q6_K: sub-blocks 2 c, 2 c + 1 are quarters (q1, q2) of half c >> 1, or (q3, q4); 16 elements to a scale.  Operands 4 (q - 32) as s8.
            const int h = c >> 1;
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {
                uint32_t A[2][2];                                  // [sub-block][row]
                float scf[2][2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint8_t* p = p0 + r * 8 * PITCH + 4 * t;
                    const uint32_t qa = word(p + 64 * h + 16 * kk), qb = word(p + 64 * h + 32 + 16 * kk), qq = word(p + 128 + 32 * h + 16 * kk);
                    if ((c & 1) == 0) {
                        A[0][r] = (((qa << 2) & 0x3C3C3C3Cu) | ((qq << 6) & 0xC0C0C0C0u)) ^ 0x80808080u;
                        A[1][r] = (((qb << 2) & 0x3C3C3C3Cu) | ((qq << 4) & 0xC0C0C0C0u)) ^ 0x80808080u;
                    } else {
                        A[0][r] = (((qa >> 2) & 0x3C3C3C3Cu) | ((qq << 2) & 0xC0C0C0C0u)) ^ 0x80808080u;
                        A[1][r] = (((qb >> 2) & 0x3C3C3C3Cu) | (qq & 0xC0C0C0C0u)) ^ 0x80808080u;
                    }
                    const uint8_t* sp = r0 + r * 8 * PITCH + 192 + 4 * c + kk;      // 16 scales in the order of the elements
                    scf[0][r] = (float)*reinterpret_cast<const int8_t*>(sp);
                    scf[1][r] = (float)*reinterpret_cast<const int8_t*>(sp + 2);
                }
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    int s12[2][4], s3[4];
                    mma16_ss0(s12[0], A[k][0], A[k][1], bw[k].a[0][kk]);
                    mma16_ss0(s12[1], A[k][0], A[k][1], bw[k].a[1][kk]);
                    mma16_ss0(s3, A[k][0], A[k][1], bw[k].b[kk]);
                    take(s12, s3, scf[k], x12[k], x3[k], a12, a3);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int r = 0; r < 2; r++) { acc12[j][r] = fmaf(d[r], a12[j][r], acc12[j][r]); acc3[j][r] = fmaf(d[r], a3[j][r], acc3[j][r]); }
}

// Shared memory: [barriers][partials: segment, tile, super-block warp, 16 rows x 8 tokens][ring: weights, tokens]
constexpr size_t R_PART = 128, R_RING = (R_PART + 2 * RTILES * RKW * 128 * 4 + 127) & ~(size_t)127;

template <int MASK>
__global__ void __launch_bounds__((RWARPS + 1) * 32, 1) gemv_rows_kernel(const __grid_constant__ RowsParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + R_STAGES;
    uint8_t* ring = smem + R_RING;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto format = [&](const RowsMat& m) { return (MASK == 1) ? 0 : (MASK == 2) ? 1 : (MASK == 4) ? 2 : (MASK == 8) ? 3 : (MASK == 16) ? 4 : m.fmt; };
    auto locate = [&](int u, int seg, int& mi, int& gl, int& pass) {
        int grp = u / p.passes;
        pass = u - grp * p.passes;
        if (p.n_seg == 2) { mi = seg; gl = grp; return; }
        mi = 0; gl = grp;
        while (mi + 1 < p.n_mat && gl >= p.mat[mi].groups) { gl -= p.mat[mi].groups; mi++; }
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) { mbar_init(full + s, 1); mbar_init(empty + s, RWARPS); }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_wait();                                                    // the tokens are the launch before's
    pdl_launch_dependents();
    const int wslot = p.slot - RKW * XB;                           // bytes of the weights in a slot
    if (warp == RWARPS) {                                          // ---- producer: a lane for each row ----
        int slot = 0, filled = 0;
        uint32_t parity = 1;
        for (int u = blockIdx.x; u < p.total_units; u += gridDim.x) {
            for (int seg = 0; seg < p.n_seg; seg++) {
                int mi, gl, pass;
                locate(u, seg, mi, gl, pass);
                const RowsMat& m = p.mat[mi];
                const int fmt = format(m), blk = fmt_bytes(fmt), row = gl * RGROUP + lane;
                const uint8_t* end = m.W + (long long)(m.out - 1) * m.pitch + (long long)p.NB * blk;
                for (int b0 = 0; b0 < p.NB; b0 += RKW) {
                    const int nb = min(RKW, p.NB - b0);
                    const uint8_t* b = m.W + (long long)row * m.pitch + (long long)b0 * blk;
                    const uint8_t* b16 = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(b) & ~(uintptr_t)15);
                    const uint8_t* e = b + nb * blk;
                    const uint8_t* e16 = reinterpret_cast<const uint8_t*>((reinterpret_cast<uintptr_t>(e) + 15) & ~(uintptr_t)15);
                    if (e16 > end) e16 -= 16;                      // what lies behind the matrix is not read: its last bytes go singly
                    const uint32_t bytes = row < m.out ? (uint32_t)(e16 - b16) : 0u;
                    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, bytes) + (uint32_t)(nb * XB);
                    if (!wait_warp(empty + slot, parity, p.status)) {
                        for (int s = 0; s < min(filled, p.stages); s++) wait_flight(full + s, s < slot ? parity ^ 1u : parity);      // the copies in flight
                        return;
                    }
                    filled = min(filled + 1, p.stages);
                    uint8_t* st = ring + (size_t)slot * p.slot;
                    uint8_t* dst = st + lane * stage_pitch(fmt, RKW);
                    if (bytes && e16 < e)
                        for (const uint8_t* q = e16; q < e; q += 2) *reinterpret_cast<uint16_t*>(dst + (q - b16)) = *reinterpret_cast<const uint16_t*>(q);
                    __syncwarp();
                    if (lane == 0) mbar_expect_tx(full + slot, total);
                    __syncwarp();
                    if (bytes) bulk_g2s(dst, b16, bytes, full + slot);
                    if (lane == 0) bulk_g2s(st + wslot, p.xr + ((size_t)pass * p.NB + b0) * XB, (uint32_t)(nb * XB), full + slot);
                    if (++slot == p.stages) { slot = 0; parity ^= 1u; }
                }
            }
        }
        return;
    }
    const int g = lane >> 2, t = lane & 3, kw = warp % RKW, tile = warp / RKW;
    float* part = reinterpret_cast<float*>(smem + R_PART) + tile * RKW * 128;       // + segment * RTILES * RKW * 128
    int slot = 0, turn = 0;
    uint32_t parity = 0;
    uint32_t tries = WAIT_TRIES;                                             // 0: a wait of this lane has run out
    for (int u = blockIdx.x; u < p.total_units; u += gridDim.x) {
        for (int seg = 0; seg < p.n_seg; seg++) {
            int mi, gl, pass;
            locate(u, seg, mi, gl, pass);
            const RowsMat& m = p.mat[mi];
            const int fmt = format(m), row = gl * RGROUP + tile * MROWS;
            float a12[2][2] = {}, a3[2][2] = {}, mins[2][2] = {};
            for (int b0 = 0; b0 < p.NB; b0 += RKW) {
                wait_phase(full + slot, parity, p.status, tries);
                if (b0 + kw < p.NB && row < m.out) {
                    const uint8_t* st = ring + (size_t)slot * p.slot;
                    const uint8_t* sb = st + tile * MROWS * stage_pitch(fmt, RKW) + kw * fmt_bytes(fmt);
                    const uint8_t* xb = st + wslot + kw * XB;
                    if ((MASK & 1) && fmt == 0) rows_block<0>(sb, 0, xb, lane, a12, a3, mins);
                    if ((MASK & 2) && fmt == 1) rows_block<1>(sb, 0, xb, lane, a12, a3, mins);
                    if ((MASK & 4) && fmt == 2) rows_block<2>(sb, (int)((uint64_t)(row + g) * (uint64_t)m.pitch + (uint32_t)(b0 * 210) & 15u), xb, lane, a12, a3, mins);
                    if ((MASK & 8) && fmt == 3) rows_block<3>(sb, 0, xb, lane, a12, a3, mins);
                    if ((MASK & 16) && fmt == 4) rows_block<4>(sb, 0, xb, lane, a12, a3, mins);
                }
                __syncwarp();
                if (lane == 0 && tries) arrive(empty + slot);
                if (++slot == p.stages) { slot = 0; parity ^= 1u; }
            }
            // (q1, q2) counted 1 / 256 of their weight; codes were carried x4 (Q6_K) or x16 (Q4_0)
            const float f3 = fmt == 2 ? 0.25f : fmt == 4 ? 1.0f / 16.0f : 1.0f, f12 = 256.0f * f3;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int r = 0; r < 2; r++) {                      // q3 of token 4 j + t sits in lane 2 j + (t >> 1) of the four, sum t & 1
                    const int src = (lane & ~3) + 2 * j + (t >> 1);
                    const float u0 = __shfl_sync(0xFFFFFFFFu, a3[0][r], src), u1 = __shfl_sync(0xFFFFFFFFu, a3[1][r], src);
                    const float v = fmaf(a12[j][r], f12, fmaf((t & 1) ? u1 : u0, f3, -mins[j][r]));
                    part[(seg * RTILES * RKW + kw) * 128 + (4 * j + t) * MROWS + g + 8 * r] = tries ? v : __uint_as_float(0x7FFFFFFFu);      // NaN
                }
        }
        named_sync<RKW * 32>(1 + tile);
        if (kw == turn) {                                          // one warp in turn adds the shares in a fixed order and applies the epilogue
            int mi, gl, pass;
            locate(u, 0, mi, gl, pass);
            const RowsMat& m = p.mat[mi];
            const int row = gl * RGROUP + tile * MROWS + (lane & 15);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int tk = 2 * i + (lane >> 4);
                float v0 = 0.f, v1 = 0.f;
#pragma unroll
                for (int w = 0; w < RKW; w++) v0 += part[w * 128 + tk * MROWS + (lane & 15)];
                if (p.n_seg == 2) {
#pragma unroll
                    for (int w = 0; w < RKW; w++) v1 += part[(RTILES * RKW + w) * 128 + tk * MROWS + (lane & 15)];
                }
                if (row < m.out && pass * 8 + tk < p.tokens) {
                    float* y = m.y + (size_t)(pass * 8 + tk) * m.out + row;
                    if (p.epilogue == GEMV_SWIGLU) *y = __fdividef(v0, 1.0f + __expf(-v0)) * v1;      // as the decode step's (gemv_kquant.cu)
                    else if (p.epilogue == GEMV_ADD) *y += v0;
                    else *y = v0;
                }
            }
        }
        named_sync<RKW * 32>(1 + tile);                            // the partials may be overwritten
        if (++turn == RKW) turn = 0;
    }
}

template <int MASK>
void launch_rows(RowsParams& p, cudaStream_t s) {
    constexpr int fmts[5] = {MASK & 1 ? 0 : -1, MASK & 2 ? 1 : -1, MASK & 4 ? 2 : -1, MASK & 8 ? 3 : -1, MASK & 16 ? 4 : -1};
    int slot = 0;
    for (int f : fmts) if (f >= 0 && RGROUP * stage_pitch(f, RKW) > slot) slot = RGROUP * stage_pitch(f, RKW);
    p.slot = slot + RKW * XB;
    p.stages = (int)((227 * 1024 - R_RING) / p.slot);
    if (p.stages > R_STAGES) p.stages = R_STAGES;
    NT_CHECK(p.stages >= 1, "gemv_rows: shared memory budget exceeded");
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(gemv_rows_kernel<MASK>, 227 * 1024, configured);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    launch_k(gemv_rows_kernel<MASK>, dim3(p.total_units < sms ? p.total_units : sms), dim3((RWARPS + 1) * 32), R_RING + (size_t)p.stages * p.slot, s, p);
    count_launch();
}

}  // namespace

size_t gemv_rows_bytes(int tokens, int K) { return (size_t)((tokens + 7) / 8) * (K / 256) * XB; }

void quantize_rows(void* xr, const float* x, const float* norm_w, float eps, int tokens, int K, cudaStream_t s) {
    NT_CHECK(K % 256 == 0 && tokens > 0, "quantize_rows: rows of whole super-blocks");
    launch_k(quantize_rows_kernel, dim3((tokens + 7) / 8 * 8), dim3(256), 0, s, static_cast<uint8_t*>(xr), x, norm_w, eps, tokens, K);
    count_launch();
}

void gemv_rows(const GemvMat* mats, int n_mat, int K, const void* xr, int tokens, GemvEpilogue ep, cudaStream_t s) {
    NT_CHECK(gemv_kq_any_pitch(mats, n_mat, K) && tokens > 0 && ep != GEMV_PEER, "gemv_rows: unsupported shape/dtype/alignment");
    NT_CHECK(ep != GEMV_SWIGLU || (n_mat == 2 && mats[0].out == mats[1].out), "gemv_rows: SWIGLU needs gate and up of equal rows");
    int mask = 0;
    for (int i = 0; i < n_mat; i++) mask |= 1 << gemv_kq_format(mats[i].dtype);
    const bool one = (mask & (mask - 1)) == 0, known = one || mask == 3 || mask == 5;
    if (!known && ep != GEMV_SWIGLU) {                             // rare mixes: one launch per matrix
        for (int i = 0; i < n_mat; i++) gemv_rows(&mats[i], 1, K, xr, tokens, ep, s);
        return;
    }
    NT_CHECK(known, "gemv_rows: SWIGLU over this format mix is not instantiated");
    RowsParams p{};
    p.n_mat = n_mat; p.NB = K / 256; p.tokens = tokens; p.passes = (tokens + 7) / 8;
    p.xr = static_cast<const uint8_t*>(xr);
    p.epilogue = (int)ep; p.n_seg = ep == GEMV_SWIGLU ? 2 : 1;
    p.status = wait_status();
    int groups = 0;
    for (int i = 0; i < n_mat; i++) {
        RowsMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W); m.y = mats[i].y; m.out = mats[i].out;
        m.groups = (m.out + RGROUP - 1) / RGROUP;
        m.fmt = gemv_kq_format(mats[i].dtype);
        m.pitch = (long long)(mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K));
        groups += m.groups;
    }
    p.total_units = (p.n_seg == 2 ? p.mat[0].groups : groups) * p.passes;
    switch (mask) {
        case 1: launch_rows<1>(p, s); break;
        case 2: launch_rows<2>(p, s); break;
        case 4: launch_rows<4>(p, s); break;
        case 3: launch_rows<3>(p, s); break;
        case 8: launch_rows<8>(p, s); break;
        case 16: launch_rows<16>(p, s); break;
        default: launch_rows<5>(p, s); break;
    }
}

}}  // namespace nt::b200
