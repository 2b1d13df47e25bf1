// gemv_mma_device.cuh — the matrix-instruction data path of the GEMV over GGUF blocks (gemv_kquant.cu): one warp multiplies 16 rows x 256-weight
// super-blocks held in shared memory by the activation vector.
//
// Activations: x[e] = xs[e / 32] * T[e] with a 24-bit integer T = q1 * 65536 + q2 * 256 + q3 (balanced digits, s8 each; |x - xs * T| <= 2^-24 of
// the 32-block's absmax), or a 32-bit one of four digits, as good as F32, where a vector was multiplied in F32 before.  mma.sync m16n8k32 with s32 accumulators multiplies the weights' 4/5/6/8-bit codes by the digits exactly: A = 16 rows
// of codes straight from the block layout, B = the digits of 32 elements.  A vector fills only three or four of B's eight columns, so B carries TWO
// groups of elements: the k positions 0-15 meet columns 0-2 (3) with group "lo", positions 16-31 meet columns 4-6 (7) with group "hi", zeros
// elsewhere.  The groups are what one byte of codes holds (low and high nibble, or the q1/q3 and q2/q4 quarters of Q6_K), so a masked word IS the
// operand, and each lane's two sums belong to one group of one row: (q1, q2) in lanes t = 0, 2, q3 (q3, q4) in lanes t = 1, 3 of a row's four.
#pragma once
#include "kernels_internal.h"
#include "ring.cuh"
#include "wait_status.cuh"
#include <cuda_fp16.h>

namespace nt { namespace b200 {
namespace {

constexpr int MROWS = 16;        // rows of one product and of a stage

__host__ __device__ constexpr int fmt_bytes(int fmt) { return fmt == 0 || fmt == 4 ? 144 : fmt == 1 ? 176 : fmt == 2 ? 210 : 272; }   // per 256 weights
// Super-blocks of a stage that KW warps share: one each; two (their chains interleave) in a team of 4 where the blocks are small.
__host__ __device__ constexpr int stage_blocks(int fmt, int KW) { return KW == 4 && fmt != 2 && fmt != 3 ? 2 * KW : KW; }
// Bytes between two rows of a stage: an odd number of 16-byte units, so that the eight rows an ldmatrix phase (16 bytes each) or a 32-bit load
// (four words each) touches lie in different banks.  Q6_K data may start 2..14 bytes into its first unit, hence one unit more.
__host__ __device__ constexpr int stage_pitch(int fmt, int KW) { return (((stage_blocks(fmt, KW) * fmt_bytes(fmt) + 15) / 16 + (fmt == 2 ? 1 : 0)) | 1) * 16; }

// The activation vector in shared memory.  Digit plane p starts at planes + p * (K + 64).  Inside a plane the four-element words are ordered so
// that a lane's words of four (Q4_K) consecutive products are one 16-byte load: element e = 64 c + 32 hi + 16 s + 4 t + i is byte i of word
// [c >> 1][hi][t][(c & 1) * 2 + s].
struct XView {
    const uint8_t* b0;          // this lane's words for columns 0-2 (3) (group lo): its plane, its t; a lane of another column points at 16 zero bytes
    const uint8_t* b1;          //   and has the offset mask 0.  b1, m1: columns 4-6 (7) (group hi)
    uint32_t m0, m1;
    const float* xs;            // [super-block][hi][4]: scale of element block 2 c + hi of the super-block, c = 0..3 (four digits: for this lane's pair)
    const float* sums;          // [super-block][8]: F32 sums of the 32-element blocks
};
__device__ __forceinline__ uint32_t xword_byte(int e) {
    return (uint32_t)((((e >> 7) * 8 + ((e >> 5) & 1) * 4 + ((e >> 2) & 3)) << 4) + ((((e >> 6) & 1) * 2 + ((e >> 4) & 1)) << 2));
}

__device__ __forceinline__ void arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
template <int N> __device__ __forceinline__ void named_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }

// Scale and integers of a 32-block of activations: x = xs * T.  amax: the largest magnitude (fmaxf: without a NaN), s: the block's sum.
//   * below 2^-126 * TOP (1e-31, 2.5e-29 for four digits) the scale would be denormal and is flushed to 0, and its reciprocal overflows: 2^-126 then, and smaller integers;
//   * a NaN (and infinities of both signs) shows in the sum and is carried by the scale, so every row's product is one;
//   * infinities are +-65537 beside zeros and the scale is infinite: the lanes of the upper and of the lower digits then multiply it by the same sum of codes, and
//     the product is an infinity of the sum's sign, or NaN where the weight is 0.  (Only for Q4_0 and Q6_K, whose vectors were F32 once; NaN for the others.)
struct BlockScale {
    float inv;
    bool infinite;
    static constexpr float TOP3 = 127.0f * 65536.0f, TOP4 = 127.0f * 16777216.0f;       // the largest integer of three and of four digits
    __device__ __forceinline__ BlockScale(float amax, float top) {
        inv = amax < top * 1.17549435e-38f ? 8.50705917e37f : __fdiv_rn(top, amax);
        infinite = amax > 3.40282347e38f;
    }
    static __device__ __forceinline__ float of(float amax, float s, float top) {       // xs
        return s != s ? s : amax < top * 1.17549435e-38f ? 1.17549435e-38f : __fdiv_rn(amax, top);
    }
    template <bool INF>                   // INF: infinities count (Q4_0, Q6_K); otherwise they are zeros under their infinite scale, NaN
    __device__ __forceinline__ void integers(const float* x, int (&T)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; i++) T[i] = __float2int_rn(__fmul_rn(x[i], inv));
        if (INF && infinite)
#pragma unroll
            for (int i = 0; i < 4; i++) T[i] = fabsf(x[i]) > 3.40282347e38f ? (x[i] > 0.f ? 65537 : -65537) : 0;
    }
};

// Balanced base-256 digits of four integers, |T| <= 127 * 65536: with 128 added to each digit they are the bytes of one sum.
__device__ __forceinline__ void digits4(const int (&T)[4], uint32_t& q1, uint32_t& q2, uint32_t& q3) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; i++) u[i] = (uint32_t)(T[i] + 0x808080);
    const uint32_t a = __byte_perm(u[0], u[1], 0x5140), b = __byte_perm(u[2], u[3], 0x5140);      // bytes 0 0 1 1
    q3 = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
    q2 = __byte_perm(a, b, 0x7632) ^ 0x80808080u;
    q1 = __byte_perm(__byte_perm(u[0], u[1], 0x0062), __byte_perm(u[2], u[3], 0x0062), 0x5410) ^ 0x80808080u;
}

// the same for four digits, |T| <= 127 * 2^24
__device__ __forceinline__ void digits4(const int (&T)[4], uint32_t& q1, uint32_t& q2, uint32_t& q3, uint32_t& q4) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; i++) u[i] = (uint32_t)T[i] + 0x80808080u;
    const uint32_t a = __byte_perm(u[0], u[1], 0x5140), b = __byte_perm(u[2], u[3], 0x5140);      // bytes 0 0 1 1
    const uint32_t c = __byte_perm(u[0], u[1], 0x7362), d = __byte_perm(u[2], u[3], 0x7362);      // bytes 2 2 3 3
    q4 = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
    q3 = __byte_perm(a, b, 0x7632) ^ 0x80808080u;
    q2 = __byte_perm(c, d, 0x5410) ^ 0x80808080u;
    q1 = __byte_perm(c, d, 0x7632) ^ 0x80808080u;
}

__device__ __forceinline__ float half_bits(uint32_t h16) { return __half2float(__ushort_as_half((unsigned short)h16)); }
// float(byte of w that sel picks) by PRMT into a 2^23 mantissa (exact)
__device__ __forceinline__ float magic_byte(uint32_t w, uint32_t sel) { return __uint_as_float(__byte_perm(w, 0x4B000000u, sel)) - 8388608.0f; }
// byte i of w, sign-extended (PRMT replicates a byte's sign where the selector's bit 3 is set)
template <int I> __device__ __forceinline__ int signed_byte(uint32_t w) {
    int d;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(w), "n"(I | (I | 8) << 4 | (I | 8) << 8 | (I | 8) << 12));
    return d;
}
__device__ __forceinline__ void mma_us(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_ss(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same onto zeros
__device__ __forceinline__ void mma_us0(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_ss0(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint4 lds128(const void* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ float sum_of(int hi, int lo) { return (float)(hi * 256 + lo); }

// What lane t's sums are multiplied by at the end: digits (q1, q2) count 256 (lanes 0, 2), q3 1 / 256 (lanes 1, 3: sum_of took it for a q1), four digits 1
// (the scales of lanes 0, 2 carry 65536); codes that the operands carry x16 (Q4_K's high nibbles, Q4_0) or x4 (Q6_K).
__device__ __forceinline__ float lane_factor(int fmt, int t, int planes) {
    const float digit = planes == 4 ? 1.0f : (t & 1) ? 1.0f / 256.0f : 256.0f;
    if (fmt == 0) return t >= 2 ? digit * (1.0f / 16.0f) : digit;
    return fmt == 2 ? digit * 0.25f : fmt == 4 ? digit * (1.0f / 16.0f) : digit;
}

// One Q6_K super-block.  ODD: the rows' data starts 2 bytes into a 4-byte word in some lane, every word is put together from two.
template <bool ODD, int PITCH>
__device__ __forceinline__ void q6_block(const uint8_t* r0, const uint8_t* b0, const uint8_t* b1, uint32_t m0, uint32_t m1, const float* xsp, int t, float (&acc)[2]) {
    const uint32_t odd = ODD ? smem_u32(r0) & 2u : 0u, sel = odd ? 0x5432u : 0x3210u;
    const uint8_t* p0 = r0 - odd + 4 * t;
    auto word = [&](const uint8_t* p) -> uint32_t {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
        return ODD ? __byte_perm(w, *reinterpret_cast<const uint32_t*>(p + 4), sel) : w;
    };
    float a[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t w0[4], w1[4];                                     // [ab][kk]
#pragma unroll
        for (int ab = 0; ab < 2; ab++) {
            const uint2 u0 = *reinterpret_cast<const uint2*>(b0 + ((h * 128 + ab * 64) & m0)), u1 = *reinterpret_cast<const uint2*>(b1 + ((h * 128 + ab * 64 + 8) & m1));
            w0[2 * ab] = u0.x; w0[2 * ab + 1] = u0.y; w1[2 * ab] = u1.x; w1[2 * ab + 1] = u1.y;
        }
        float v[2][2][2];                                          // [kk][ab][row]
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
            uint32_t lo[2][2], hi[2][2];                           // [row][ab]
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint8_t* p = p0 + r * 8 * PITCH;
                const uint32_t qa = word(p + 64 * h + 16 * kk), qb = word(p + 64 * h + 32 + 16 * kk), qq = word(p + 128 + 32 * h + 16 * kk);
                lo[r][0] = (((qa << 2) & 0x3C3C3C3Cu) | ((qq << 6) & 0xC0C0C0C0u)) ^ 0x80808080u;
                lo[r][1] = (((qb << 2) & 0x3C3C3C3Cu) | ((qq << 4) & 0xC0C0C0C0u)) ^ 0x80808080u;
                hi[r][0] = (((qa >> 2) & 0x3C3C3C3Cu) | ((qq << 2) & 0xC0C0C0C0u)) ^ 0x80808080u;
                hi[r][1] = (((qb >> 2) & 0x3C3C3C3Cu) | (qq & 0xC0C0C0C0u)) ^ 0x80808080u;
            }
#pragma unroll
            for (int ab = 0; ab < 2; ab++) {
                int s[4];
                mma_ss0(s, lo[0][ab], lo[1][ab], hi[0][ab], hi[1][ab], w0[2 * ab + kk], w1[2 * ab + kk]);
                v[kk][ab][0] = sum_of(s[0], s[1]); v[kk][ab][1] = sum_of(s[2], s[3]);
            }
        }
        const float x0 = xsp[2 * h + (t >> 1)], x1 = xsp[4 + 2 * h + (t >> 1)];
#pragma unroll
        for (int r = 0; r < 2; r++) {                              // the scales' bytes 2 ab + kk
            const uint32_t sc = word(p0 + r * 8 * PITCH + 192 + 8 * h + 4 * (t >> 1) - 4 * t);
            a[r] = fmaf(x0, fmaf(v[0][0][r], (float)signed_byte<0>(sc), v[1][0][r] * (float)signed_byte<1>(sc)), a[r]);
            a[r] = fmaf(x1, fmaf(v[0][1][r], (float)signed_byte<2>(sc), v[1][1][r] * (float)signed_byte<3>(sc)), a[r]);
        }
    }
    acc[0] = fmaf(half_bits(*reinterpret_cast<const uint16_t*>(r0 + 208)), a[0], acc[0]);
    acc[1] = fmaf(half_bits(*reinterpret_cast<const uint16_t*>(r0 + 8 * PITCH + 208)), a[1], acc[1]);
}

// acc[0] (row g) and acc[1] (row g + 8) += the lane's share of the product of N super-blocks (sb: the first in row 0 of the stage, sbi its index in
// the vector; the next ones KW further on), to be scaled by lane_factor; mins += what the offsets subtract (Q4_K, Q5_K; not scaled).
// mis: bytes between the row slot's first unit and row g's data (Q6_K; the same 8 rows on).
template <int FMT, int N, int KW>
__device__ __forceinline__ void tile_blocks(const uint8_t* sb, int mis, int sbi, const XView& xv, int lane, float (&acc)[2], float (&mins)[2]) {
    constexpr int PITCH = stage_pitch(FMT, KW), NEXT = KW * fmt_bytes(FMT);
    const int g = lane >> 2, t = lane & 3;
    const uint8_t* b0 = xv.b0 + ((uint32_t)(sbi * 256) & xv.m0);
    const uint8_t* b1 = xv.b1 + ((uint32_t)(sbi * 256) & xv.m1);
    const float* xsp = xv.xs + sbi * 8;
    if (FMT <= 1) {
        // ---- Q4_K / Q5_K: [d, dmin][12 bytes of 6-bit scales and mins]([32 bytes of fifth bits])[128 bytes of nibbles] ----
        const uint32_t msel = 0x7440u + 2 * (t & 1), ssel = 0x7440u + (t >> 1);
        const uint32_t ad = smem_u32(sb) + (uint32_t)((lane & 15) * PITCH + (lane >> 4) * 16);
        float a[N][2], d[N][2], xs[N][4];
        uint32_t sc[N][2][2], qh[N][4];
#pragma unroll
        for (int n = 0; n < N; n++) {
            const float4 x4 = *reinterpret_cast<const float4*>(xsp + n * KW * 8 + (t >> 1) * 4);
            xs[n][0] = x4.x; xs[n][1] = x4.y; xs[n][2] = x4.z; xs[n][3] = x4.w;
            const float2 sums = *reinterpret_cast<const float2*>(xv.sums + sbi * 8 + n * KW * 8 + 2 * t);
            if (FMT == 1) ldsm4(qh[n], ad + n * NEXT + 16);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint4 h = lds128(sb + n * NEXT + (g + 8 * r) * PITCH);
                sc[n][r][0] = h.y & 0x3F3F3F3Fu;
                sc[n][r][1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
                const uint32_t m = t < 2 ? h.z & 0x3F3F3F3Fu : ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
                mins[r] = fmaf(half_bits(h.x >> 16), fmaf(magic_byte(m, msel), sums.x, magic_byte(m, msel + 1) * sums.y), mins[r]);
                d[n][r] = half_bits(h.x & 0xFFFFu);
                a[n][r] = 0.f;
            }
        }
#pragma unroll
        for (int cc = 0; cc < 2; cc++) {
#pragma unroll
            for (int n = 0; n < N; n++) {
                const uint4 v0 = lds128(b0 + ((n * KW * 256 + cc * 128) & xv.m0)), v1 = lds128(b1 + ((n * KW * 256 + cc * 128 + 64) & xv.m1));
                const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int ch = 2 * cc + c;
                    const float x23 = -8388608.0f * xs[n][ch];     // scale * x = (2^23 + scale) * x - 2^23 * x, rounded once
                    uint32_t q[4], lo[4], hi[4];
                    ldsm4(q, ad + n * NEXT + (FMT == 0 ? 16 : 48) + 32 * ch);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        lo[i] = q[i] & 0x0F0F0F0Fu;
                        if (FMT == 0) {
                            hi[i] = q[i] & 0xF0F0F0F0u;            // codes x16, u8
                        } else {
                            lo[i] |= ((ch < 2 ? qh[n][i] << (4 - 2 * ch) : qh[n][i] >> (2 * ch - 4))) & 0x10101010u;
                            hi[i] = ((q[i] >> 4) & 0x0F0F0F0Fu) | (((ch < 2 ? qh[n][i] << (3 - 2 * ch) : qh[n][i] >> (2 * ch - 3))) & 0x10101010u);
                        }
                    }
                    int s[4];
                    mma_us0(s, lo[0], lo[1], hi[0], hi[1], w0[2 * c], w1[2 * c]);
                    mma_us(s, lo[2], lo[3], hi[2], hi[3], w0[2 * c + 1], w1[2 * c + 1]);
#pragma unroll
                    for (int r = 0; r < 2; r++)
                        a[n][r] = fmaf(sum_of(s[2 * r], s[2 * r + 1]), fmaf(__uint_as_float(__byte_perm(sc[n][r][cc], 0x4B000000u, ssel + 2 * c)), xs[n][ch], x23), a[n][r]);
                }
            }
        }
#pragma unroll
        for (int n = 0; n < N; n++) {
            acc[0] = fmaf(d[n][0], a[n][0], acc[0]);
            acc[1] = fmaf(d[n][1], a[n][1], acc[1]);
        }
    } else if (FMT == 2) {
        // ---- Q6_K: [128 bytes of low nibbles][64 bytes of high pairs][16 s8 scales][d]; 210 bytes, so data starts at any even address.
        // The operands are 4 (q - 32) as s8: the six bits moved to the top of the byte, the top bit flipped. ----
        const uint8_t* r0 = sb + g * PITCH + mis;
        if (__any_sync(0xFFFFFFFFu, smem_u32(r0) & 2u)) q6_block<true, PITCH>(r0, b0, b1, xv.m0, xv.m1, xsp, t, acc);
        else q6_block<false, PITCH>(r0, b0, b1, xv.m0, xv.m1, xsp, t, acc);
    } else {
        // ---- Q8_0 (eight blocks of [d][32 x s8], 34 bytes) and Q4_0 ([d][16 bytes of nibbles], 18 bytes): pairs of blocks, the first of a pair has
        // its codes 2 bytes into a word, the second on a word ----
        constexpr int B = FMT == 3 ? 34 : 18;
#pragma unroll
        for (int cc = 0; cc < 2; cc++) {
#pragma unroll
            for (int n = 0; n < N; n++) {
                const uint4 v0 = lds128(b0 + ((n * KW * 256 + cc * 128) & xv.m0)), v1 = lds128(b1 + ((n * KW * 256 + cc * 128 + 64) & xv.m1));
                const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
                const float2 x2 = *reinterpret_cast<const float2*>(xsp + n * KW * 8 + (t >> 1) * 4 + 2 * cc);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const uint8_t* p = sb + n * NEXT + g * PITCH + 2 * B * (2 * cc + c);
                    auto first = [&](const uint8_t* a) { return __byte_perm(*reinterpret_cast<const uint32_t*>(a), *reinterpret_cast<const uint32_t*>(a + 4), 0x5432u); };
                    auto second = [&](const uint8_t* a) { return *reinterpret_cast<const uint32_t*>(a + B + 2); };
                    int s[4];
                    const uint8_t* a = p + 4 * t;
                    if (FMT == 3) {
                        mma_ss0(s, first(a), first(a + 8 * PITCH), second(a), second(a + 8 * PITCH), w0[2 * c], w1[2 * c]);
                        a += 16;
                        mma_ss(s, first(a), first(a + 8 * PITCH), second(a), second(a + 8 * PITCH), w0[2 * c + 1], w1[2 * c + 1]);
                    } else {
                        const uint32_t f0 = first(a), f1 = first(a + 8 * PITCH), n0 = second(a), n1 = second(a + 8 * PITCH);
                        auto lo = [](uint32_t q) { return ((q << 4) & 0xF0F0F0F0u) ^ 0x80808080u; };     // 16 (q - 8) as s8
                        auto hi = [](uint32_t q) { return (q & 0xF0F0F0F0u) ^ 0x80808080u; };
                        mma_ss0(s, lo(f0), lo(f1), hi(f0), hi(f1), w0[2 * c], w0[2 * c + 1]);
                        mma_ss(s, lo(n0), lo(n1), hi(n0), hi(n1), w1[2 * c], w1[2 * c + 1]);
                    }
#pragma unroll
                    for (int r = 0; r < 2; r++)
                        acc[r] = fmaf(sum_of(s[2 * r], s[2 * r + 1]) * (c ? x2.y : x2.x), half_bits(*reinterpret_cast<const uint16_t*>(p + B * (t >> 1) + r * 8 * PITCH)), acc[r]);
                }
            }
        }
    }
}

}  // namespace
}}  // namespace nt::b200
