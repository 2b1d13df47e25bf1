// prefill_blocks.cu — tensor-core GEMM of several tokens over matrices in GGUF blocks: Y[T, N] (+)= X[T, K] . W[N, K]^T, W expanded on the way to the MMA.
//
// The reference has no batched product (prefill loops its GEMV over the tokens, src/model/attention.cpp:144-162, ffn.cpp:96-133).  Here a CTA owns 128 rows of W
// and NT tokens:
//   * the roles of the operands are exchanged: W is A (M = 128 rows), tokens are B (N = NT, a multiple of 16 up to 128);
//   * A holds INTEGERS.  A weight of Q4_K is d * (sc * q) - dmin * m, of Q5_K the same: sc * q <= 63 * 31 is exact in F16, so one F16 operand carries the weight
//     and d joins when the epilogue takes a super-block's sum out of tensor memory.  The minima are a product of their own, m (8 for a super-block) times the sums
//     of 32 activations.  Q6_K's sc * (q - 32) has up to 14 bits: a pair of halves, the second -1, 0 or 1.  Q8_0 and Q4_0 have a scale for 32 weights: d_i * q as
//     a pair of halves, exact, under a power of two for the super-block;
//   * eight warps (Q6_K: twelve) expand 64 columns of 128 rows at a time, a row to a lane: blocks come into shared memory by TMA (Q6_K rows off 16 bytes by cp.async), two halves cost a PRMT and an HFMA2,
//     and go to TENSOR MEMORY, from where tcgen05.mma takes its A operand: shared memory's bandwidth is left to B;
//   * B is the split of the tokens x = hi + lo by TMA: two products for 16 columns (hi, lo), a third with the low half of a pair; in the fine form x = hi + lo + third,
//     as many bits as the 24-bit integers hold and more (three products, five with a pair);
//   * a super-block (256 columns; half of one where a row has no more, 64 where the caller asks for it) to an accumulator: the tensor cores cut off each addition, which leaves 1.86e-8 of a sum for
//     each.  The epilogue's eight warps add the sums in F32 registers, times d, and write C once;
//   * the work, tiles times super-blocks, is dealt out evenly: a CTA takes a run of super-blocks, whichever tiles it touches.  A tile that several CTAs share goes
//     to a scratch, and whoever comes last adds the shares in their order (nothing waits for another CTA, the sums do not depend on who was last).
// Measured (gate and up of an 8B layer, 28672 x 4096 Q4_K; the form before, which expanded each weight to a pair of halves, beside it): 500 tokens 341 -> 218 us, with 61 %
// of the tensor cycles and 41 bytes a clock and SM from L2, where 128 x 128 tiles with two halves of each token ask for 64 at full rate; 21 tokens 100 (24-bit integers,
// three passes) -> 57 us, and 43 in the form for a few tokens below.
#include "kernels_internal.h"
#include "ring.cuh"
#include "tc_device.cuh"
#include "wait_status.cuh"
#include "gemv_mma_device.cuh"
#include "tile_deal.cuh"
#include <cuda.h>
#include <cuda_fp16.h>
#include <algorithm>

namespace nt { namespace b200 {

namespace {

constexpr int QBK = 64;                                  // columns of a k-block: a 128-byte swizzle row of F16
constexpr int NT_MAX = 128, FEW_TOKENS = 32;             // tokens of a tile; of a launch of the form for a few
constexpr int STAGES_MAX = 4, D_BUFS_MAX = 4, RAW_MAX = 8, SCALE_RING = 8;
constexpr int EXP_WARP = 12;      // warp 0 tokens, 1 MMA, 2 blocks (2, 3: off 16 bytes), 4-11 epilogue, from 12 on expansion
// Warps of expansion that share 32 rows, k-blocks in turn.  Three where the expansion is what bounds: Q6_K (500 tokens, 4096 x 14336: 178 us with two, 160), and pairs of halves over few
// tokens (21, 28672 x 4096: Q6_K 71.5, 67.2; Q8_0 63.6, 61.0); products or waits bound the others (Q8_0, 500 tokens 299, 308; Q4_K over few 44.0, 44.3), and formats side by side have
// no registers for it.  No more of them than stages: a warp waits for the k-block a ring before its own, and knows of the one before that only as long as its last one is no older.
__host__ __device__ constexpr int groups(int mask) { return mask == 4 ? 3 : 2; }
__host__ __device__ constexpr int few_groups(int mask) { return mask == 4 || mask == 8 || mask == 16 ? 3 : 2; }
__host__ __device__ constexpr int threads(int groups) { return (EXP_WARP + 4 * groups) * 32; }

// Bytes between rows of a super-block in shared memory: an odd number of 16-byte units.  Q6_K lies at any even address: the units around it.
__host__ __device__ constexpr int raw_pitch(int fmt) { return fmt == 2 ? 240 : fmt_bytes(fmt); }
__host__ __device__ constexpr bool has_mins(int fmt) { return fmt <= 1; }      // otherwise A is a pair of halves

struct alignas(64) BlkMaps { CUtensorMap x, sums, w[3]; };      // tokens, their sums, matrices as 32-bit words
struct BlkParams : Deal {
    int Mp, kc, stages, b_stage, raw_depth, raw_slot, a_cols, d_bufs;
    int d_cols;                // the form for a few tokens: columns of a stage's sums
    int tma;                   // a matrix's rows come by TMA (bits)
    unsigned* status;          // wait_status.cuh
};

__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&v)[4]) {      // the four words twice
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// K-major rows of 32 bytes under SWIZZLE_32B: eight rows are 256 bytes (make_desc's layout with type 6)
__device__ __forceinline__ uint64_t make_desc32(const void* smem_ptr) {
    const uint64_t addr = (uint64_t)(smem_u32(smem_ptr) & 0x3FFFFu) >> 4;
    return addr | (1ull << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}
// Q6_K rows that do not lie 16 bytes apart, which TMA does not take: 64 rows of super-block b into a slot by units, four lanes to a row.  Rows behind the matrix are
// its last one, and nothing behind the matrix's end is read.
__device__ __forceinline__ void copy_rows(uint32_t slot, const DealMat& m, int row, int b, int NB, int lane) {
    constexpr int PITCH = raw_pitch(2), UNITS = 14;
    const uint8_t* end = m.W + (long long)(m.rows - 1) * m.pitch + (long long)NB * fmt_bytes(2);
#pragma unroll 2
    for (int r = lane >> 2; r < 64; r += 8) {
        const uint8_t* p = m.W + (long long)min(row + r, m.rows - 1) * m.pitch + (long long)b * fmt_bytes(2);
        p = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)15);
        const int left = (int)min((long long)(end - p), 256ll);
#pragma unroll
        for (int i = 0; i < (UNITS + 3) / 4; i++) {
            const int u = 4 * i + (lane & 3), n = min(16, left - 16 * u);
            if (u < UNITS && n > 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot + r * PITCH + 16 * u), "l"(p + 16 * u), "r"(n) : "memory");
        }
    }
}

__device__ __forceinline__ __half2 h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// bytes i, j of w as halves 1024 + byte
template <int I, int J> __device__ __forceinline__ __half2 half_pair(uint32_t w) { return h2(__byte_perm(w, 0x64646464u, 0x4040u | I | (J << 8))); }
__device__ __forceinline__ __half2 half_twice(uint32_t w, int i) { return h2(__byte_perm(w, 0x64646464u, 0x4040u + 0x0101u * i)); }

// The scales and minima of a Q4_K / Q5_K super-block as bytes: sub-blocks 0-3 or 4-7
__device__ __forceinline__ uint32_t kq_scales(const uint4& h, bool upper) { return upper ? (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu; }
__device__ __forceinline__ uint32_t kq_mins(const uint4& h, bool upper) { return upper ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu; }

// k-block c (64 columns) of a Q4_K / Q5_K super-block: sc * q, two columns to a word
template <int FMT>
__device__ __forceinline__ void expand_k(const uint8_t* blk, const uint4& h, int c, uint32_t (&out)[32]) {
    const uint4 a = lds128(blk + (FMT == 0 ? 16 : 48) + 32 * c), b = lds128(blk + (FMT == 0 ? 32 : 64) + 32 * c);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t v[8];
    if (FMT == 1) {
        const uint4 e = lds128(blk + 16), f = lds128(blk + 32);
        const uint32_t u[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = u[i] >> (2 * c);        // bits 0 and 1: the fifth bits of the two sub-blocks
    }
    const uint32_t ss = kq_scales(h, c >= 2);
    const __half2 k = __float2half2_rn(1024.0f), neg = __float2half2_rn(-1024.0f);
#pragma unroll
    for (int s = 0; s < 2; s++) {
        const __half2 sc = __hsub2(half_twice(ss, 2 * (c & 1) + s), k), off = __hmul2(sc, neg);      // -1024 sc: exact, up to 64512
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint32_t q = (s ? w[i] >> 4 : w[i]) & 0x0F0F0F0Fu;
            if (FMT == 1) q |= (s ? v[i] << 3 : v[i] << 4) & 0x10101010u;
            out[16 * s + 2 * i] = bits(__hfma2(half_pair<0, 1>(q), sc, off));
            out[16 * s + 2 * i + 1] = bits(__hfma2(half_pair<2, 3>(q), sc, off));
        }
    }
}

// N words from any even address, by whole units (32-bit loads of rows an odd number of units apart would meet four to a bank)
template <int N> __device__ __forceinline__ void lds_words(const uint8_t* p, uint32_t (&w)[N]) {
    constexpr int UNITS = (N + 7) / 4;
    const uint32_t at = smem_u32(p), sel = (at & 2u) ? 0x5432u : 0x3210u;
    const uint8_t* a = p - (at & 15u);
    uint32_t u[4 * UNITS];
#pragma unroll
    for (int i = 0; i < UNITS; i++) { const uint4 v = lds128(a + 16 * i); u[4 * i] = v.x; u[4 * i + 1] = v.y; u[4 * i + 2] = v.z; u[4 * i + 3] = v.w; }
#pragma unroll
    for (int i = 0; i < N + 2; i++) u[i] = (at & 8u) ? u[i + 2] : u[i];
#pragma unroll
    for (int i = 0; i < N + 1; i++) u[i] = (at & 4u) ? u[i + 1] : u[i];
#pragma unroll
    for (int i = 0; i < N; i++) w[i] = __byte_perm(u[i], u[i + 1], sel);
}
// Half hf of k-block c of the other formats as pairs of halves.  codes: what has to be taken off 1024 + code; D: the scale of the first and the second 16 columns
__device__ __forceinline__ void pairs(const uint32_t (&q)[8], __half2 off, const __half2 (&D)[2], uint32_t (&hi)[16], uint32_t (&lo)[16]) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const __half2 v = __hsub2(j ? half_pair<2, 3>(q[i]) : half_pair<0, 1>(q[i]), off), p = __hmul2_rn(v, D[i >> 2]);
            hi[2 * i + j] = bits(p);
            lo[2 * i + j] = bits(__hfma2(v, D[i >> 2], __hneg2(p)));      // what the product's rounding left, exact
        }
}
// Q6_K: the upper bits of a k-block's codes, the same words for its two halves
__device__ __forceinline__ void upper_bits(const uint8_t* blk, int c, uint32_t (&v)[8]) { lds_words(blk + 128 + 32 * (c >> 1), v); }
template <int FMT>
__device__ __forceinline__ void expand_pair(const uint8_t* blk, int c, int hf, float up, const uint32_t (&v)[8], uint32_t (&hi)[16], uint32_t (&lo)[16]) {
    uint32_t q[8];
    __half2 D[2];
    if (FMT == 2) {
        // half h of the super-block, quarters q1 (codes in the low nibbles of the first 32 bytes, bits 0-1 of the pairs), q2 (second 32, bits 2-3), q3, q4
        const int h = c >> 1, qt = 2 * (c & 1) + hf;
        uint32_t w[8];
        lds_words(blk + 64 * h + 32 * hf, w);
        const int8_t* sc = reinterpret_cast<const int8_t*>(blk + 192 + 8 * h + 2 * qt);
        D[0] = __half2half2(__int2half_rn(sc[0])); D[1] = __half2half2(__int2half_rn(sc[1]));
#pragma unroll
        for (int i = 0; i < 8; i++) {                              // bits 4 and 5 from the word whose bits 2 qt and 2 qt + 1 they are
            const uint32_t a = w[i] >> (4 * (c & 1)), b = __funnelshift_l(v[i], v[i], 36 - 2 * qt);      // (what comes round is masked off)
            q[i] = ((a & 0x0F0F0F0Fu) | (b & ~0x0F0F0F0Fu)) & 0x3F3F3F3Fu;
        }
        pairs(q, __float2half2_rn(1056.0f), D, hi, lo);
    } else {
        const uint8_t* b = blk + (FMT == 3 ? 34 : 18) * (2 * c + hf);
        D[0] = D[1] = __float2half2_rn(half_bits(*reinterpret_cast<const uint16_t*>(b)) * up);
        if (FMT == 3) {
            lds_words(b + 2, q);
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] ^= 0x80808080u;
        } else {
            uint32_t w[4];
            lds_words(b + 2, w);
#pragma unroll
            for (int i = 0; i < 4; i++) { q[i] = w[i] & 0x0F0F0F0Fu; q[4 + i] = (w[i] >> 4) & 0x0F0F0F0Fu; }
        }
        pairs(q, __float2half2_rn(FMT == 3 ? 1152.0f : 1032.0f), D, hi, lo);
    }
}
// Q8_0, Q4_0: the power of two that takes a super-block's largest scale to 16 .. 32 (the product's low half then lies far above the least F16 number), and its
// inverse.  Scales that are zero, or not finite: 1.
template <int FMT>
__device__ __forceinline__ float block_power(const uint8_t* blk, float& inverse) {
    int e = 0;
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) top = max(top, (uint32_t)*reinterpret_cast<const uint16_t*>(blk + (FMT == 3 ? 34 : 18) * i) & 0x7FFFu);
    if (top && top < 0x7C00u) e = (int)(__float_as_uint(half_bits(top)) >> 23) - 127 - 4;
    inverse = __uint_as_float((uint32_t)(127 + e) << 23);
    return __uint_as_float((uint32_t)(127 - e) << 23);
}

template <int MASK> __device__ __forceinline__ int format(int fmt) { return MASK == 1 ? 0 : MASK == 2 ? 1 : MASK == 4 ? 2 : MASK == 8 ? 3 : MASK == 16 ? 4 : fmt; }
template <int MASK> __device__ __forceinline__ bool mins_of(const BlkParams& p, int mi) { return (MASK & (MASK - 1)) == 0 ? (MASK & 3) != 0 : (MASK & 3) != 0 && has_mins(p.mat[mi].fmt); }

// One thread, or (Q6_K rows off 16 bytes) both warps of the producer: blocks of W, the 16-byte units around a super-block of 128 rows, by TMA or by cp.async
template <int MASK>
__device__ __forceinline__ void load_blocks(const BlkMaps& maps, const BlkParams& p, int u0, int u1, uint8_t* raw, uint64_t* raw_full, uint64_t* raw_empty, bool by_tma, uint32_t dead, int warp, int lane) {
    uint32_t st = 0, par = 1, filled = 0;
    Place q = start(p, u0);
    for (int u = u0; u < u1; u++, next(p, q)) {
        const DealMat& m = p.mat[q.mi];
        const int fmt = format<MASK>(m.fmt);
        wait_cta(raw_empty + st, par, dead);
        if (word_set(dead)) {
            for (uint32_t s = 0; s < filled && by_tma; s++) wait_flight(raw_full + s, s < st ? par ^ 1u : par);      // the copies in flight
            break;
        }
        filled = min(filled + 1, (uint32_t)p.raw_depth);
        uint8_t* d = raw + (size_t)st * p.raw_slot;
        if (by_tma || (p.tma >> q.mi & 1)) {
            if (threadIdx.x == 64) {
                mbar_expect_tx(raw_full + st, 128u * raw_pitch(fmt));
                tma_load_2d(d, &maps.w[q.mi], (q.b * fmt_bytes(fmt) & ~15) >> 2, q.row0, raw_full + st);
            }
            if (!by_tma) mbar_arrive(raw_full + st);
        } else {
            copy_rows(smem_u32(d) + (warp - 2) * 64 * raw_pitch(2), m, q.row0 + (warp - 2) * 64, q.b, p.NB, lane);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(raw_full + st)) : "memory");
            if (threadIdx.x == 64) mbar_arrive(raw_full + st);
        }
        if (++st == (uint32_t)p.raw_depth) { st = 0; par ^= 1; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The super-block that this lane's row has in a slot, the power of two that its codes are taken up by and its inverse; what its sums and its minima's sum are multiplied by
template <int MASK>
__device__ __forceinline__ const uint8_t* find_block(const DealMat& m, const Place& q, int fmt, const uint8_t* slot, int r, float& up, float& down) {
    const uint8_t* blk = slot + r * raw_pitch(fmt);
    if ((MASK & 4) && fmt == 2) blk += ((uint32_t)min(q.row0 + r, m.rows - 1) * (uint32_t)m.pitch + (uint32_t)q.b * 210u) & 15u;      // (W on 16 bytes)
    up = down = 1.f;
    if ((MASK & 8) && fmt == 3) up = block_power<3>(blk, down);
    if ((MASK & 16) && fmt == 4) up = block_power<4>(blk, down);
    return blk;
}
template <int MASK>
__device__ __forceinline__ float2 block_scale(const uint8_t* blk, int fmt, float down) {
    float2 s = make_float2(down, 0.f);
    if ((MASK & 3) && fmt <= 1) { const uint32_t h = *reinterpret_cast<const uint32_t*>(blk); s = make_float2(half_bits(h & 0xFFFFu), -32.0f * half_bits(h >> 16)); }
    if ((MASK & 4) && fmt == 2) s.x = half_bits(*reinterpret_cast<const uint16_t*>(blk + 208));
    return s;
}
// the minima of a Q4_K / Q5_K super-block as halves
__device__ __forceinline__ void expand_mins(const uint4& h, uint32_t (&w)[4]) {
    const __half2 k = __float2half2_rn(1024.0f);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t mm = kq_mins(h, i != 0);
        w[2 * i] = bits(__hsub2(half_pair<0, 1>(mm), k));
        w[2 * i + 1] = bits(__hsub2(half_pair<2, 3>(mm), k));
    }
}

// MASK: the formats that a launch's matrices have (bits).  PARTS: halves that a token's column is split into
template <int MASK, int PARTS>
__global__ void __launch_bounds__(threads(groups(MASK)), 1) gemm_blocks_kernel(const __grid_constant__ BlkMaps maps, const __grid_constant__ BlkParams p) {
    constexpr bool ONE = (MASK & (MASK - 1)) == 0, MINS = (MASK & 3) != 0, PAIRS = (MASK & 28) != 0;
    constexpr int XG = groups(MASK);                            // warps of expansion that share 32 rows
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // a stage is a k-block of the tokens (shared memory) and of W (tensor memory) under one pair of barriers
    __shared__ uint64_t full[STAGES_MAX], empty[STAGES_MAX], d_full[D_BUFS_MAX], d_empty[D_BUFS_MAX];
    __shared__ uint64_t raw_full[RAW_MAX], raw_empty[RAW_MAX], s_full[SCALE_RING];
    __shared__ float2 scales[SCALE_RING][128];                     // of a super-block's rows: what its sum and what its minima's sum are multiplied by
    __shared__ uint32_t tmem_base_smem, last_smem, dead_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NT = p.NT;
    const uint32_t b_tile = (uint32_t)NT * 128, b_stage = (uint32_t)p.b_stage, dead = smem_u32(&dead_smem);
    uint8_t* raw = smem + (size_t)p.stages * b_stage;
    const int u0 = first_unit(p, blockIdx.x), u1 = first_unit(p, blockIdx.x + 1);      // this CTA's super-blocks
    const bool by_tma = !(MASK & 4) || p.tma == (1 << p.n_mat) - 1;      // all of W
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.stages; i++) { mbar_init(full + i, 5); mbar_init(empty + i, 1); }      // the tokens' producer and four warps of the expansion
        for (int i = 0; i < p.d_bufs; i++) { mbar_init(d_full + i, 1); mbar_init(d_empty + i, 8); }
        for (int i = 0; i < p.raw_depth; i++) { mbar_init(raw_full + i, by_tma ? 1 : 65); mbar_init(raw_empty + i, 4 * XG); }
        for (int i = 0; i < SCALE_RING; i++) mbar_init(s_full + i, 4);
        dead_smem = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // Weights depend on no launch in flight: their copies and expansion start at once, tokens and everything written wait for the launch before
    pdl_launch_dependents();
    // tensor memory is this CTA's whole (its address is 0): sums, expanded k-blocks, minima
    const uint32_t a_base = (uint32_t)(p.d_bufs * NT), m_base = a_base + (uint32_t)(p.stages * p.a_cols);

    // registers: 640 threads x 96 at launch; 56 + 2 x 120 + 2 x 88 for the five warpgroups are no more (six with 80: 48 + 2 x 96 + 3 x 80)
    if (warp < EPI_WARP) {
    if constexpr (XG == 3) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
        if (lane == 0) {                                           // ---- tokens by TMA ----
            uint32_t st = 0, par = 1, filled = 0;
            Place q = start(p, u0);
            pdl_wait();
            for (int u = u0; u < u1; u++, next(p, q)) {
                const bool mins = mins_of<MASK>(p, q.mi);
                for (int kb = 0; kb < 4; kb++) {
                    wait_cta(empty + st, par, dead);
                    if (word_set(dead)) {
                        for (uint32_t s = 0; s < filled; s++) wait_flight(full + s, s < st ? par ^ 1u : par);      // the copies in flight
                        u = u1;
                        break;
                    }
                    filled = min(filled + 1, (uint32_t)p.stages);
                    uint8_t* d = smem + (size_t)st * b_stage;
                    mbar_expect_tx(full + st, PARTS * b_tile + (mins && kb == 3 ? (PARTS - 1) * NT * 32u : 0u));
#pragma unroll
                    for (int i = 0; i < PARTS; i++) tma_load_2d(d + i * b_tile, &maps.x, q.b * 256 + kb * QBK, i * p.Mp + q.t0, full + st);      // a part lies Mp rows below the one before
                    if (mins && kb == 3)
#pragma unroll
                        for (int i = 0; i < PARTS - 1; i++) tma_load_2d(d + PARTS * b_tile + i * NT * 32, &maps.sums, q.b * 16, i * p.Mp + q.t0, full + st);
                    if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA: the whole warp walks the loop, so that addresses and descriptors stay in uniform registers, and one lane issues (a loop of lane 0
        // alone moved every operand of every MMA there: about 100 cycles an instruction) ----
        const uint32_t lead = elect_lane();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | (8u << 24);      // D F32, A and B F16 K-major, N, M = 128
        const uint64_t desc0 = make_desc(smem), desc32 = make_desc32(smem), lo_step = (uint64_t)(b_tile >> 4), stage_step = (uint64_t)(b_stage >> 4);
        uint32_t st = 0, par = 0, db = 0, dpar = 1;
        int last = -1;                                             // stage and parity of the last commit
        Place q = start(p, u0);
        for (int u = u0; u < u1; u++, next(p, q)) {
            const bool mins = mins_of<MASK>(p, q.mi);
#pragma unroll 1
            for (int k0 = 0; k0 < 4; k0 += p.kc) {
                wait_cta(d_empty + db, dpar, dead);
                const uint32_t d = db * NT;
#pragma unroll 1
                for (int kb = k0; kb < k0 + p.kc; kb++) {
                    wait_cta(full + st, par, dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bh = desc0 + st * stage_step, bl = bh + lo_step;
                    const uint32_t ah = a_base + st * p.a_cols, al = ah + 32;
                    uint32_t acc = kb != k0;
                    auto product = [&](uint32_t a, uint64_t b) {
                        umma_ts_by(lead, d, a, b, idesc, acc);
#pragma unroll
                        for (int k = 1; k < 4; k++) umma_ts_by(lead, d, a + 8 * k, b + 2 * k, idesc, 1u);
                        acc = 1u;
                    };
                    // the small products first (what is left out is 2^-22 of a product with two parts, 2^-33 with three)
                    if (PARTS == 3) {
                        if (PAIRS && (ONE || !mins)) product(al, bl);
                        product(ah, bl + lo_step);
                    }
                    if (PAIRS && (ONE || !mins)) product(al, bh);
                    product(ah, bl);
                    product(ah, bh);
                    last = (int)(st * 2 + par);
                    if (kb == 3 && mins) break;                    // its stage is free after the minima
                    umma_commit_by(lead, empty + st);
                    if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                }
                umma_commit_by(lead, d_full + db);
                if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
            }
            if (MINS && mins) {                                    // minima: 8 of them times the halves of 8 sums, twice (the third halves, and zeros, before)
                wait_cta(d_empty + db, dpar, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t sums = desc32 + st * stage_step + PARTS * lo_step;
                if (PARTS == 3) umma_ts_by(lead, db * NT, m_base, sums + (NT * 32 >> 4), idesc, 0u);
                umma_ts_by(lead, db * NT, m_base, sums, idesc, PARTS == 3);
                umma_commit_by(lead, empty + st);                  // (the minima's place is free with this stage)
                umma_commit_by(lead, d_full + db);
                if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
                if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
            }
        }
        if (word_set(dead) && last >= 0) wait_flight(empty + (last >> 1), last & 1);      // given up: the products in flight
    } else if (by_tma ? threadIdx.x == 64 : true) {
        load_blocks<MASK>(maps, p, u0, u1, raw, raw_full, raw_empty, by_tma, dead, warp, lane);      // ---- blocks of W ----
    }
    } else if (warp < EXP_WARP) {
        if constexpr (XG == 3) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        else asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
        // ---- epilogue: a lane is a row of W; two warps share a quarter's rows, every other 16 tokens to each ----
        const int quarter = warp & 3, half = (warp - EPI_WARP) >> 2, r = quarter * 32 + lane;
        const uint32_t tq = ((uint32_t)(quarter * 32) << 16) + half * 16;
        uint32_t db = 0, dpar = 0, slot = 0, spar = 0;
        Place q = start(p, u0);
        pdl_wait();
        const float* token_scale = behind_wait(p.scale);
        for (int u = u0; u < u1;) {
            const int sums = 4 / p.kc, chunks = sums + (MINS && mins_of<MASK>(p, q.mi) ? 1 : 0);
            const int seg0 = u, end = min(u1, u + (p.NB - q.b));
            uint64_t acc[4][8] = {};                               // pairs of tokens
#pragma unroll 1
            for (; u < end; u++) {
                wait_cta(s_full + slot, spar, dead);
                const float2 s = scales[slot][r];
                if (++slot == SCALE_RING) { slot = 0; spar ^= 1; }
#pragma unroll 1
                for (int c = 0; c < chunks; c++) {
                    const float f = c == sums ? s.y : s.x;
                    const uint64_t ff = pack2(f, f);
                    wait_cta(d_full + db, dpar, dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (32 * i + 16 * half >= NT) break;
                        uint32_t v[16];
                        tmem_ld16(tq + db * NT + 32 * i, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 8; j++) acc[i][j] = fma2(pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), ff, acc[i][j]);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty + db);
                    if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
                }
            }
            finish_tile<4, 32>(p, q, acc, u0, seg0, end, 16 * half, r, token_scale, &last_smem, dead);
            q.b = 0; q.tile++;
            place(p, q);
        }
        if (word_set(dead)) report(p.status);
    } else {                                                       // ---- expansion: two warps share 32 rows; k-blocks 0, 2 or 1, 3 of a super-block to each ----
        if constexpr (XG == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        const int quarter = warp & 3, group = (warp - EXP_WARP) >> 2;
        const uint32_t tq = (uint32_t)(quarter * 32) << 16;
        int slot = 0, sslot = 0;
        uint32_t st = group, par = 1, rpar = 0;
        auto wrap = [&] { if (st >= (uint32_t)p.stages) { st -= p.stages; par ^= 1; } };      // (stages >= XG)
        wrap();
        int first = group;                                         // of this warp's k-blocks in a super-block: every XG-th of the run is its
        Place q = start(p, u0);
        for (int u = u0; u < u1; u++, next(p, q)) {
            const DealMat& m = p.mat[q.mi];
            const int fmt = format<MASK>(m.fmt);
            wait_cta(raw_full + slot, rpar, dead);
            float up, down;
            const uint8_t* blk = find_block<MASK>(m, q, fmt, raw + (size_t)slot * p.raw_slot, quarter * 32 + lane, up, down);
            if (group == 0) {
                scales[sslot][quarter * 32 + lane] = block_scale<MASK>(blk, fmt, down);
                __syncwarp();
                if (lane == 0) mbar_arrive(s_full + sslot);
            }
            if (++sslot == SCALE_RING) sslot = 0;
#pragma unroll 1
            for (int c = XG == 2 ? group : first; c < 4; c += XG) {
                const uint32_t a = tq + a_base + st * p.a_cols;
                if (MINS && fmt <= 1) {
                    uint32_t v[32];
                    const uint4 h = lds128(blk);
                    if ((MASK & 1) && fmt == 0) expand_k<0>(blk, h, c, v);
                    if ((MASK & 2) && fmt == 1) expand_k<1>(blk, h, c, v);
                    wait_cta(empty + st, par, dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    tmem_st16(a, v);
                    tmem_st16(a + 16, v + 16);
                    if (c == 3) {                                  // (the product of the minima before came ahead of the commit that freed a stage of k-block 3 or later)
                        uint32_t w[4];
                        expand_mins(h, w);
                        tmem_st8(tq + m_base, w);
                    }
                } else if (PAIRS) {
                    uint32_t v[8];
                    if (MASK == 4) upper_bits(blk, c, v);
#pragma unroll 1
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t hi[16], lo[16];
                        if (MASK != 4 && (MASK & 4) && fmt == 2) upper_bits(blk, c, v);      // (formats side by side have no registers to keep them)
                        if ((MASK & 4) && fmt == 2) expand_pair<2>(blk, c, hf, up, v, hi, lo);
                        if ((MASK & 8) && fmt == 3) expand_pair<3>(blk, c, hf, up, v, hi, lo);
                        if ((MASK & 16) && fmt == 4) expand_pair<4>(blk, c, hf, up, v, hi, lo);
                        if (hf == 0) {
                            wait_cta(empty + st, par, dead);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        tmem_st16(a + 16 * hf, hi);
                        tmem_st16(a + 32 + 16 * hf, lo);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full + st);
                st += XG;
                wrap();
            }
            if (XG == 3) first = first == 0 ? 2 : first - 1;
            if (lane == 0) mbar_arrive(raw_empty + slot);          // (every lane has read what it stored)
            if (++slot == p.raw_depth) { slot = 0; rpar ^= 1; }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_smem), "n"(512));
}

// The same for up to 32 tokens in the fine form (64 columns to an accumulator, a token in three halves).  There the products take a fifth of a k-block's time, memory a sixth: what
// bounds is that copies, expansion, products and sums hand each k-block on by barriers, two commits and five waits of a warp to each (the MMA warp's wait for a free accumulator
// alone took 270 of 1050 cycles).  So a stage is half a super-block, with accumulators of its own, and one barrier (done) says that its products are finished, which frees its
// tokens and weights and hands its sums over.  A super-block of Q4_K takes 2200 cycles where it took 3200; the expansion's instructions bound then, of Q6_K above all (5000).
// 21 tokens, us with the split of the tokens, before and now: Q4_K 28672 x 4096 56.6, 43.1; 4096 x 14336 39.1, 31.1; 4096 x 4096 21.2, 18.3; Q5_K 14336 x 4096 37.1, 29.8; Q6_K
// 4096 x 14336 48.5, 46.2, and 43.7 with twelve warps of expansion.  Sixteen warps of expansion and four of sums in place of eight and eight: 57.6 (the four are then behind, and the issuing warp is starved).
// Tiles of more than 32 tokens leave room for one stage of it: 40 tokens 60.8, 70.8.
template <int MASK>
__global__ void __launch_bounds__(threads(few_groups(MASK)), 1) gemm_blocks_few_kernel(const __grid_constant__ BlkMaps maps, const __grid_constant__ BlkParams p) {
    constexpr bool ONE = (MASK & (MASK - 1)) == 0, MINS = (MASK & 3) != 0, PAIRS = (MASK & 28) != 0;
    // Q8_0, Q4_0: a super-block's sums are added up by themselves first, which keeps small what small numbers are added to (14336 columns, error 1.54e-7 -> 1.39e-7, as gemv_rows')
    constexpr bool APART = MASK == 8 || MASK == 16;
    constexpr int XG = few_groups(MASK);                            // warps of expansion that share 32 rows
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[STAGES_MAX], done[STAGES_MAX], d_empty[STAGES_MAX];
    __shared__ uint64_t raw_full[RAW_MAX], raw_empty[RAW_MAX], s_full[SCALE_RING];
    __shared__ float2 scales[SCALE_RING][128];
    __shared__ uint32_t tmem_base_smem, last_smem, dead_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NT = p.NT;
    const uint32_t b_tile = (uint32_t)NT * 128, b_stage = (uint32_t)p.b_stage, dead = smem_u32(&dead_smem);
    uint8_t* raw = smem + (size_t)p.stages * b_stage;
    const int u0 = first_unit(p, blockIdx.x), u1 = first_unit(p, blockIdx.x + 1);
    const bool by_tma = !(MASK & 4) || p.tma == (1 << p.n_mat) - 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.stages; i++) { mbar_init(full + i, 9); mbar_init(done + i, 1); mbar_init(d_empty + i, 8); }      // the tokens' producer and eight warps of the expansion
        for (int i = 0; i < p.raw_depth; i++) { mbar_init(raw_full + i, by_tma ? 1 : 65); mbar_init(raw_empty + i, 4 * XG); }
        for (int i = 0; i < SCALE_RING; i++) mbar_init(s_full + i, 4);
        dead_smem = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_launch_dependents();
    // tensor memory, stage by stage: sums (two k-blocks; minima where a matrix of the launch has them), expanded k-blocks, minima.  Laid out by the host alone: formats side by
    // side have one kernel, whether any of them has minima or none
    const uint32_t d_cols = (uint32_t)p.d_cols, a_base = (uint32_t)p.stages * d_cols, m_base = a_base + (uint32_t)(p.stages * 2 * p.a_cols);

    if (warp < EPI_WARP) {
    if constexpr (XG == 3) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
        if (lane == 0) {                                           // ---- tokens by TMA ----
            uint32_t st = 0, par = 1, filled = 0;
            Place q = start(p, u0);
            pdl_wait();
            for (int u = u0; u < u1; u++, next(p, q)) {
                const bool mins = mins_of<MASK>(p, q.mi);
                for (int h = 0; h < 2; h++) {
                    wait_cta(done + st, par, dead);
                    if (word_set(dead)) {
                        for (uint32_t s = 0; s < filled; s++) wait_flight(full + s, s < st ? par ^ 1u : par);      // the copies in flight
                        u = u1;
                        break;
                    }
                    filled = min(filled + 1, (uint32_t)p.stages);
                    uint8_t* d = smem + (size_t)st * b_stage;
                    mbar_expect_tx(full + st, 6 * b_tile + (mins && h ? 64u * NT : 0u));
#pragma unroll
                    for (int i = 0; i < 6; i++) tma_load_2d(d + i * b_tile, &maps.x, q.b * 256 + (2 * h + i / 3) * QBK, (i % 3) * p.Mp + q.t0, full + st);      // a part lies Mp rows below the one before
                    if (mins && h)
#pragma unroll
                        for (int i = 0; i < 2; i++) tma_load_2d(d + 6 * b_tile + i * NT * 32, &maps.sums, q.b * 16, i * p.Mp + q.t0, full + st);
                    if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA: the whole warp walks the loop, one lane issues ----
        const uint32_t lead = elect_lane();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | (8u << 24);
        const uint64_t desc0 = make_desc(smem), desc32 = make_desc32(smem), part_step = (uint64_t)(b_tile >> 4), stage_step = (uint64_t)(b_stage >> 4);
        uint32_t st = 0, par = 0;
        int last = -1;
        Place q = start(p, u0);
        for (int u = u0; u < u1; u++, next(p, q)) {
            const bool mins = mins_of<MASK>(p, q.mi);
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                wait_cta(d_empty + st, par ^ 1u, dead);
                wait_cta(full + st, par, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t b0 = desc0 + st * stage_step;
                const uint32_t d0 = st * d_cols, a0 = a_base + st * 2 * p.a_cols;
#pragma unroll 1
                for (int kb = 0; kb < 2; kb++) {
                    const uint64_t bh = b0 + 3 * kb * part_step, bl = bh + part_step, b3 = bl + part_step;
                    const uint32_t d = d0 + kb * NT, ah = a0 + kb * p.a_cols, al = ah + 32;
                    uint32_t acc = 0u;
                    auto product = [&](uint32_t a, uint64_t b) {
                        umma_ts_by(lead, d, a, b, idesc, acc);
#pragma unroll
                        for (int k = 1; k < 4; k++) umma_ts_by(lead, d, a + 8 * k, b + 2 * k, idesc, 1u);
                        acc = 1u;
                    };
                    // the small products first (what is left out is 2^-33 of a product)
                    if (PAIRS && (ONE || !mins)) product(al, bl);
                    product(ah, b3);
                    if (PAIRS && (ONE || !mins)) product(al, bh);
                    product(ah, bl);
                    product(ah, bh);
                }
                if (MINS && mins && h) {                           // minima: 8 of them times the halves of 8 sums, twice (the third halves, and zeros, before)
                    const uint64_t sums = desc32 + st * stage_step + 6 * part_step;
                    umma_ts_by(lead, d0 + 2 * NT, m_base + 8 * st, sums + (NT * 32 >> 4), idesc, 0u);
                    umma_ts_by(lead, d0 + 2 * NT, m_base + 8 * st, sums, idesc, 1u);
                }
                umma_commit_by(lead, done + st);
                last = (int)(st * 2 + par);
                if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
            }
        }
        if (word_set(dead) && last >= 0) wait_flight(done + (last >> 1), last & 1);      // given up: the products in flight
    } else if (by_tma ? threadIdx.x == 64 : true) {
        load_blocks<MASK>(maps, p, u0, u1, raw, raw_full, raw_empty, by_tma, dead, warp, lane);      // ---- blocks of W ----
    }
    } else if (warp < EXP_WARP) {
        if constexpr (XG == 3) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        else asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
        // ---- epilogue: a lane is a row of W; two warps share a quarter's rows, 16 tokens to each ----
        const int quarter = warp & 3, half = (warp - EPI_WARP) >> 2, r = quarter * 32 + lane;
        const uint32_t tq = ((uint32_t)(quarter * 32) << 16) + half * 16;
        uint32_t st = 0, par = 0, slot = 0, spar = 0;
        Place q = start(p, u0);
        pdl_wait();
        const float* token_scale = behind_wait(p.scale);
        for (int u = u0; u < u1;) {
            const bool mins = mins_of<MASK>(p, q.mi);
            const int seg0 = u, end = min(u1, u + (p.NB - q.b));
            uint64_t acc[1][8] = {};                               // pairs of tokens
#pragma unroll 1
            for (; u < end; u++) {
                wait_cta(s_full + slot, spar, dead);
                const float2 s = scales[slot][r];
                const uint64_t fx = pack2(s.x, s.x), fy = pack2(s.y, s.y), one = pack2(1.f, 1.f);
                uint64_t sum[8] = {};
                if (++slot == SCALE_RING) { slot = 0; spar ^= 1; }
#pragma unroll 1
                for (int h = 0; h < 2; h++) {
                    wait_cta(done + st, par, dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (16 * half < NT) {
                        uint32_t v[2][16], m[16];
                        const uint32_t d = tq + st * d_cols;
                        tmem_ld16(d, v[0]);
                        tmem_ld16(d + NT, v[1]);
                        if (MINS && mins && h) tmem_ld16(d + 2 * NT, m);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 2; i++)
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                const uint64_t x = pack2(__uint_as_float(v[i][2 * j]), __uint_as_float(v[i][2 * j + 1]));
                                if (APART) sum[j] = fma2(x, one, sum[j]);
                                else acc[0][j] = fma2(x, fx, acc[0][j]);
                            }
                        if (APART && h)
#pragma unroll
                            for (int j = 0; j < 8; j++) acc[0][j] = fma2(sum[j], fx, acc[0][j]);
                        if (MINS && mins && h)
#pragma unroll
                            for (int j = 0; j < 8; j++) acc[0][j] = fma2(pack2(__uint_as_float(m[2 * j]), __uint_as_float(m[2 * j + 1])), fy, acc[0][j]);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty + st);
                    if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                }
            }
            finish_tile<1, 32>(p, q, acc, u0, seg0, end, 16 * half, r, token_scale, &last_smem, dead);
            q.b = 0; q.tile++;
            place(p, q);
        }
        if (word_set(dead)) report(p.status);
    } else {                                                       // ---- expansion: two warps share 32 rows; a k-block of a stage to each ----
        if constexpr (XG == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        const int quarter = warp & 3, group = (warp - EXP_WARP) >> 2;
        const uint32_t tq = (uint32_t)(quarter * 32) << 16;
        int slot = 0, sslot = 0;
        uint32_t st = group >> 1, par = 1, rpar = 0;              // (two stages and more)
        int first = group;                                         // of this warp's k-blocks in a super-block: every XG-th of the run is its
        Place q = start(p, u0);
        for (int u = u0; u < u1; u++, next(p, q)) {
            const DealMat& m = p.mat[q.mi];
            const int fmt = format<MASK>(m.fmt);
            wait_cta(raw_full + slot, rpar, dead);
            float up, down;
            const uint8_t* blk = find_block<MASK>(m, q, fmt, raw + (size_t)slot * p.raw_slot, quarter * 32 + lane, up, down);
            if (group == 0) {
                scales[sslot][quarter * 32 + lane] = block_scale<MASK>(blk, fmt, down);
                __syncwarp();
                if (lane == 0) mbar_arrive(s_full + sslot);
            }
            if (++sslot == SCALE_RING) sslot = 0;
#pragma unroll 1
            for (int c = XG == 2 ? group : first; c < 4; c += XG) {
                const uint32_t a = tq + a_base + (2 * st + (c & 1)) * p.a_cols;
                if (MINS && fmt <= 1) {
                    uint32_t v[32];
                    const uint4 h = lds128(blk);
                    if ((MASK & 1) && fmt == 0) expand_k<0>(blk, h, c, v);
                    if ((MASK & 2) && fmt == 1) expand_k<1>(blk, h, c, v);
                    wait_cta(done + st, par, dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    tmem_st16(a, v);
                    tmem_st16(a + 16, v + 16);
                    if (c == 3) {
                        uint32_t w[4];
                        expand_mins(h, w);
                        tmem_st8(tq + m_base + 8 * st, w);
                    }
                } else if (PAIRS) {
                    uint32_t v[8];
                    if (MASK == 4) upper_bits(blk, c, v);
#pragma unroll 1
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t hi[16], lo[16];
                        if (MASK != 4 && (MASK & 4) && fmt == 2) upper_bits(blk, c, v);      // (formats side by side have no registers to keep them)
                        if ((MASK & 4) && fmt == 2) expand_pair<2>(blk, c, hf, up, v, hi, lo);
                        if ((MASK & 8) && fmt == 3) expand_pair<3>(blk, c, hf, up, v, hi, lo);
                        if ((MASK & 16) && fmt == 4) expand_pair<4>(blk, c, hf, up, v, hi, lo);
                        if (hf == 0) {
                            wait_cta(done + st, par, dead);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        tmem_st16(a + 16 * hf, hi);
                        tmem_st16(a + 32 + 16 * hf, lo);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full + st);
                st += XG == 2 ? 1 : 1 + (c & 1);
                if (st >= (uint32_t)p.stages) { st -= p.stages; par ^= 1; }
            }
            if (XG == 3) first = first == 0 ? 2 : first - 1;
            if (lane == 0) mbar_arrive(raw_empty + slot);          // (every lane has read what it stored)
            if (++slot == p.raw_depth) { slot = 0; rpar ^= 1; }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_smem), "n"(512));
}

// ---- tokens ----
// One block to a token: x (MODE 1: RMSNorm(x) * w, rmsnorm.cu:17-70's math; 2: silu(x) * w, gemm.cu:713-725's expression; 3: hi x and lo w of
// a plain split, which may be the one written to) as F16 hi + lo, the sums of 32 of them
// (a 32nd part, so that they stay within F16) as hi + lo, FINE: the halves that those two leave of both, and the factor that undoes the token's power of two.  That power takes the largest to 2^13 .. 2^14, where the
// low halves keep their bits.  Block 0 also clears the product's counts: a launch whose wait ran out leaves some behind.
// TOK_NORM_ANY: TOK_NORM whose gains do not lie on 16 bytes.  BF16 parts: no power; those for dense matrices: no sums.
enum : int { TOK_PLAIN = 0, TOK_NORM = 1, TOK_SILU = 2, TOK_SPLIT = 3, TOK_NORM_ANY = 4 };
template <int MODE, bool FINE, TokenParts PARTS>
__global__ void __launch_bounds__(512) split_tokens_kernel(__half* hi, __half* lo, __half* third, __half* __restrict__ sums, __half* __restrict__ third_sums, float* __restrict__ scale, unsigned* __restrict__ count, int counts,
                                                           const float* xin, const float* w, float eps, int K) {
    constexpr bool BF16 = PARTS == TokenParts::BF16;
    constexpr int KEEP = 7;                                        // chunks of 2048 held in registers: rows to 14336
    __shared__ float red[2][16];
    const int tid = threadIdx.x;
    pdl_wait();
    pdl_launch_dependents();               // after the wait: the product reads weights before its own, and whatever wrote them came before this launch
    if (blockIdx.x == 0) for (int i = tid; i < counts; i += 512) count[i] = 0;
    const size_t at = (size_t)blockIdx.x * K;
    const float* x = xin + at;
    const float* y = MODE == TOK_SILU ? w + at : w;
    auto value = [&](int i, float& ss) {                           // before the norm's factor
        if (MODE == TOK_SPLIT) {
            const uint2 a = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(xin) + at + i), b = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(w) + at + i);
            const float2 a0 = __half22float2(h2(a.x)), a1 = __half22float2(h2(a.y)), b0 = __half22float2(h2(b.x)), b1 = __half22float2(h2(b.y));
            return make_float4(a0.x + b0.x, a0.y + b0.y, a1.x + b1.x, a1.y + b1.y);
        }
        float4 a = *reinterpret_cast<const float4*>(x + i);
        if (MODE == TOK_NORM || MODE == TOK_NORM_ANY) {
            const float4 g = MODE == TOK_NORM ? *reinterpret_cast<const float4*>(y + i) : make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
            ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
            a.x *= g.x; a.y *= g.y; a.z *= g.z; a.w *= g.w;
        }
        if (MODE == TOK_SILU) {
            const float4 u = *reinterpret_cast<const float4*>(y + i);
            auto f = [](float p, float q) { return p / (1.0f + expf(-p)) * q; };
            a = make_float4(f(a.x, u.x), f(a.y, u.y), f(a.z, u.z), f(a.w, u.w));
        }
        return a;
    };
    float4 keep[KEEP];
    float ss = 0.f, amax = 0.f, none = 0.f;
    auto most = [&](const float4& a) { amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)))); };
#pragma unroll
    for (int c = 0; c < KEEP; c++) { const int i = c * 2048 + 4 * tid; if (i < K) { keep[c] = value(i, ss); most(keep[c]); } }
    for (int i = KEEP * 2048 + 4 * tid; i < K; i += 2048) most(value(i, ss));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o); amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o)); }
    if ((tid & 31) == 0) { red[0][tid >> 5] = ss; red[1][tid >> 5] = amax; }
    __syncthreads();
    float tot = 0.f, f = 1.f;
#pragma unroll
    for (int i = 0; i < 16; i++) { tot += red[0][i]; amax = fmaxf(amax, red[1][i]); }
    if (MODE == TOK_NORM || MODE == TOK_NORM_ANY) f = rsqrtf(tot / K + eps);
    const uint32_t e = __float_as_uint(amax * f) >> 23 & 255u;     // not finite, or zero: as it is
    const uint32_t up = BF16 || e == 255u || e == 0u ? 127u : min(227u, max(27u, 267u - e));
    f *= __uint_as_float(up << 23);
    if (tid == 0) scale[blockIdx.x] = __uint_as_float((254u - up) << 23);
    __half* h = hi + (size_t)blockIdx.x * K;
    __half* l = lo + (size_t)blockIdx.x * K;
    const size_t sm = (size_t)blockIdx.x * (K / 16);
    auto rest = [](float v, uint32_t h, uint32_t l, bool upper) {  // what two halves leave of v: exact
        if (BF16) return upper ? v - __uint_as_float(h & 0xFFFF0000u) - __uint_as_float(l & 0xFFFF0000u) : v - __uint_as_float(h << 16) - __uint_as_float(l << 16);
        const float2 fh = __half22float2(h2(h)), fl = __half22float2(h2(l));
        return upper ? v - fh.y - fl.y : v - fh.x - fl.x;
    };
    [[maybe_unused]] auto pair = [](float a, float b) { uint32_t h, l; split_pair(a, b, BF16, h, l); return h; };
    auto split = [](float a, float b, uint32_t& h, uint32_t& l) {
        if (PARTS != TokenParts::F16_SHORT) { split_pair(a, b, BF16, h, l); return; }
        // the nearest numbers of 24 - n bits, c = 2^n + 1 (Dekker's splitting)
        auto top = [](float a, float b, float c) { const float p = __fmul_rn(a, c), q = __fmul_rn(b, c); return __floats2half2_rn(__fsub_rn(p, __fsub_rn(p, a)), __fsub_rn(q, __fsub_rn(q, b))); };
        const __half2 p = top(a, b, 1048577.0f);
        const float2 f = __half22float2(p);
        h = bits(p); l = bits(top(a - f.x, b - f.y, 65537.0f));
    };
    auto put = [&](int i, float4 a) {
        a.x *= f; a.y *= f; a.z *= f; a.w *= f;
        uint2 ph, pl;
        split(a.x, a.y, ph.x, pl.x);
        split(a.z, a.w, ph.y, pl.y);
        *reinterpret_cast<uint2*>(h + i) = ph;
        *reinterpret_cast<uint2*>(l + i) = pl;
        if (FINE)
            *reinterpret_cast<uint2*>(third + (size_t)blockIdx.x * K + i) =
                make_uint2(pair(rest(a.x, ph.x, pl.x, false), rest(a.y, ph.x, pl.x, true)), pair(rest(a.z, ph.y, pl.y, false), rest(a.w, ph.y, pl.y, true)));
        if (PARTS != TokenParts::F16) return;                      // (dense matrices have no minima)
        float s = (a.x + a.y) + (a.z + a.w);                       // K is a multiple of 256: whole warps
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 1); s += __shfl_xor_sync(0xFFFFFFFFu, s, 2); s += __shfl_xor_sync(0xFFFFFFFFu, s, 4);
        if ((tid & 7) == 0) {
            s *= 1.0f / 32.0f;
            const __half sh = __float2half_rn(s);
            const float left = s - __half2float(sh);
            const __half sl = __float2half_rn(left);
            const size_t q = sm + (i >> 8) * 16 + ((i >> 5) & 7);
            sums[q] = sh; sums[q + 8] = sl;
            if (FINE) { third_sums[q] = __float2half_rn(left - __half2float(sl)); third_sums[q + 8] = __float2half_rn(0.f); }
        }
    };
#pragma unroll
    for (int c = 0; c < KEEP; c++) { const int i = c * 2048 + 4 * tid; if (i < K) put(i, keep[c]); }
    for (int i = KEEP * 2048 + 4 * tid; i < K; i += 2048) put(i, value(i, none));
}
__global__ void __launch_bounds__(512) plain_tokens_kernel(float* __restrict__ scale, int rows, unsigned* __restrict__ count, int counts) {
    pdl_wait();
    pdl_launch_dependents();               // after the wait, as above
    for (int i = threadIdx.x; i < rows; i += 512) scale[i] = 1.0f;
    for (int i = threadIdx.x; i < counts; i += 512) count[i] = 0;
}
// silu(g) * u (gemm.cu:713-725's expression) straight into the split of the next product
__global__ void __launch_bounds__(256) silu_split_kernel(uint2* __restrict__ hi, uint2* __restrict__ lo, const float4* __restrict__ g, const float4* __restrict__ u, size_t n4) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const float4 a = g[i], b = u[i];
    auto f = [](float x, float y) { return x / (1.0f + expf(-x)) * y; };
    uint2 h, l;
    split_pair(f(a.x, b.x), f(a.y, b.y), 0, h.x, l.x);
    split_pair(f(a.z, b.z), f(a.w, b.w), 0, h.y, l.y);
    hi[i] = h; lo[i] = l;
}

template <int MASK>
void launch_blocks(const BlkMaps& maps, const BlkParams& p, int parts, bool few, int grid, size_t smem, cudaStream_t s) {
    static unsigned long long configured[3] = {};      // bit per device id
    auto launch = [&](auto kernel, int groups, unsigned long long& done) {
        opt_in_dynamic_smem(kernel, 214 * 1024, done);
        launch_k_pdl(true, kernel, dim3(grid), dim3(threads(groups)), smem, s, maps, p);
    };
    if (few) launch(gemm_blocks_few_kernel<MASK>, few_groups(MASK), configured[0]);
    else if (parts == 3) launch(gemm_blocks_kernel<MASK, 3>, groups(MASK), configured[1]);
    else launch(gemm_blocks_kernel<MASK, 2>, groups(MASK), configured[2]);
    count_launch();
}

size_t padded(int T) { return ((size_t)T + 127) / 128 * 128; }
int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}

}  // namespace

bool gemm_blocks_supported(const GemvMat* mats, int n_mat, int K) { return gemv_kq_any_pitch(mats, n_mat, K); }

// [hi rows][lo rows][third rows][their sums, part by part: fine has three, two of sums][scales][counts], rows padded to 128.  The front is gemm_f16_tc_workspace_bytes.
static size_t parts_bytes(int T, int K, bool fine) { return gemm_f16_tc_workspace_bytes(T, K) / 2 * (fine ? 3 : 2); }
static size_t sums_bytes(int T, int K, bool fine) { return padded(T) * ((size_t)K / 8) * (fine ? 2 : 1); }
size_t block_tokens_bytes(int T, int K, bool fine) { return parts_bytes(T, K, fine) + sums_bytes(T, K, fine) + padded(T) * sizeof(float) + (size_t)sm_count() * sizeof(unsigned); }
// tokens of a tile, as even as they come
static int tile_tokens(int T) { const int cols = (T + NT_MAX - 1) / NT_MAX; return ((T + cols - 1) / cols + 15) / 16 * 16; }
size_t block_scratch_bytes(int T) { return (size_t)sm_count() * 2 * 128 * (T > NT_MAX ? NT_MAX : tile_tokens(T)) * sizeof(float); }

BlockTokens block_tokens(void* workspace, int T, int K, bool fine) {
    BlockTokens t;
    uint8_t* p = static_cast<uint8_t*>(workspace);
    t.split = p;
    t.sums = p + parts_bytes(T, K, fine);
    t.scale = reinterpret_cast<float*>(p + parts_bytes(T, K, fine) + sums_bytes(T, K, fine));
    t.count = reinterpret_cast<unsigned*>(t.scale + padded(T));
    t.fine = fine;
    return t;
}

namespace {
template <int MODE>
BlockTokens launch_split(void* workspace, const float* x, const float* w, float eps, int T, int K, bool fine, TokenParts parts, cudaStream_t s) {
    const BlockTokens t = block_tokens(workspace, T, K, fine);
    const size_t part = padded(T) * (size_t)K;
    __half *hi = static_cast<__half*>(t.split), *sums = static_cast<__half*>(t.sums);
    const auto kernel = parts == TokenParts::BF16 ? (fine ? split_tokens_kernel<MODE, true, TokenParts::BF16> : split_tokens_kernel<MODE, false, TokenParts::BF16>)
                        : !fine                   ? split_tokens_kernel<MODE, false, TokenParts::F16>
                        : parts == TokenParts::F16 ? split_tokens_kernel<MODE, true, TokenParts::F16> : split_tokens_kernel<MODE, true, TokenParts::F16_SHORT>;
    launch_k_pdl(true, kernel, dim3(T), dim3(512), 0, s, hi, hi + part, hi + 2 * part, sums, sums + part / 16, t.scale, t.count, sm_count(), x, w, eps, K);
    count_launch();
    return t;
}
}  // namespace

BlockTokens split_tokens(void* workspace, const float* x, const float* norm_w, float eps, int T, int K, bool fine, cudaStream_t s, TokenParts parts) {
    if (!norm_w) return launch_split<TOK_PLAIN>(workspace, x, nullptr, 0.f, T, K, fine, parts, s);
    return (reinterpret_cast<uintptr_t>(norm_w) & 15) ? launch_split<TOK_NORM_ANY>(workspace, x, norm_w, eps, T, K, fine, parts, s) : launch_split<TOK_NORM>(workspace, x, norm_w, eps, T, K, fine, parts, s);
}
BlockTokens silu_split_tokens(void* workspace, const float* gate, const float* up, int T, int K, bool fine, cudaStream_t s, TokenParts parts) {
    return launch_split<TOK_SILU>(workspace, gate, up, 0.f, T, K, fine, parts, s);
}
BlockTokens resplit_tokens(void* workspace, const void* hi, const void* lo, int T, int K, cudaStream_t s) {
    return launch_split<TOK_SPLIT>(workspace, static_cast<const float*>(hi), static_cast<const float*>(lo), 0.f, T, K, false, TokenParts::F16, s);
}
// A plain split as it lies, for matrices without minima: it has no sums, and powers of 2^0
static size_t plain_tokens_bytes(int T) { return padded(T) * sizeof(float) + (size_t)sm_count() * sizeof(unsigned); }
static BlockTokens plain_tokens(void* memory, const void* split, int T, cudaStream_t s) {
    BlockTokens t;
    t.split = t.sums = const_cast<void*>(split);
    t.scale = static_cast<float*>(memory);
    t.count = reinterpret_cast<unsigned*>(t.scale + padded(T));
    launch_k_pdl(true, plain_tokens_kernel, dim3(1), dim3(512), 0, s, t.scale, (int)padded(T), t.count, sm_count());
    count_launch();
    return t;
}

bool gemm_blocks_for_few(const GemvMat* mats, int n_mat, int K, int tokens) {
    bool pairs = true;
    long long weights = 0;
    for (int i = 0; i < n_mat; i++) {
        pairs = pairs && (mats[i].dtype == DType::Q8_0 || mats[i].dtype == DType::Q4_0);
        weights += (long long)mats[i].out * K;
    }
    return tokens > (pairs && weights <= 8 << 20 ? 16 : 8);
}

bool gemm_blocks(const GemvMat* mats, int n_mat, int K, const BlockTokens& x, void* scratch, int T, bool add, cudaStream_t s) {
    if (T <= 0 || !gemm_blocks_supported(mats, n_mat, K)) return false;
    const int sms = sm_count();
    BlkParams p{};
    p.status = wait_status();
    p.n_mat = n_mat; p.T = T; p.NB = K / 256; p.add = add;
    p.Mp = (int)padded(T);
    p.scale = x.scale; p.alpha = 1.0f;
    p.kc = x.fine ? 1 : p.NB == 1 ? 2 : 4;
    const int parts = x.fine ? 3 : 2;
    const bool few = x.fine && T <= FEW_TOKENS;
    int tiles = 0, slot = 0, mask = 0;
    for (int i = 0; i < n_mat; i++) {
        DealMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W); m.C = mats[i].y; m.rows = mats[i].out; m.tiles = (m.rows + 127) / 128;
        m.fmt = gemv_kq_format(mats[i].dtype);
        m.pitch = (long long)(mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K));
        tiles += m.tiles;
        slot = std::max(slot, 128 * raw_pitch(m.fmt));
        mask |= 1 << m.fmt;
    }
    const bool mins = mask & 3, pairs = mask & 28;
    p.cols = (T + NT_MAX - 1) / NT_MAX;
    p.NT = tile_tokens(T);
    p.units = tiles * p.cols * p.NB;
    // tensor memory: buffers of sums, expanded k-blocks, 8 columns of minima.  Shared memory: the same stages of tokens, and blocks of W behind them (the deeper the
    // fewer tokens there are: weights from HBM are then what bounds)
    p.a_cols = pairs ? 64 : 32;
    p.raw_slot = slot;
    const size_t cap = 213 * 1024;
    if (few) {                                                     // a stage is two k-blocks, with sums of its own
        p.d_cols = (mins ? 3 : 2) * p.NT;
        p.b_stage = (p.NT * (6 * 128 + (mins ? 64 : 0)) + 1023) / 1024 * 1024;
        p.stages = std::min(STAGES_MAX, 512 / (p.d_cols + 2 * p.a_cols + (mins ? 8 : 0)));
    } else {
        p.b_stage = (p.NT * (128 * parts + (mins ? 32 * (parts - 1) : 0)) + 1023) / 1024 * 1024;
        for (p.stages = STAGES_MAX; p.stages > 2; p.stages--) {
            p.d_bufs = std::min(D_BUFS_MAX, (512 - p.stages * p.a_cols - (mins ? 8 : 0)) / p.NT);
            if (p.d_bufs >= (mins ? 3 : 2) && (size_t)p.stages * p.b_stage + 2 * (size_t)slot <= cap) break;
        }
        p.d_bufs = std::min(D_BUFS_MAX, (512 - p.stages * p.a_cols - (mins ? 8 : 0)) / p.NT);
        if (p.d_bufs < 2 || p.stages < groups(mask)) return false;      // (the latter: 3 with tiles of 128 tokens in three parts, otherwise 4)
    }
    p.raw_depth = (int)std::min<size_t>(RAW_MAX, (cap - (size_t)p.stages * p.b_stage) / slot);
    if (p.raw_depth < 1) return false;
    const int grid = std::min(sms, p.units);
    p.part = static_cast<float*>(scratch);
    p.count = x.count;
    BlkMaps maps;
    if (!tc_map_f16(&maps.x, x.split, parts * (uint64_t)p.Mp, (uint64_t)K, (uint32_t)p.NT) ||
        !tc_map_f16_rows32(&maps.sums, x.sums, (parts - 1) * (uint64_t)p.Mp, (uint64_t)K / 16, (uint32_t)p.NT))
        return false;
    for (int i = 0; i < n_mat; i++) {
        const DealMat& m = p.mat[i];
        if (m.pitch & 15) continue;
        if (!tc_map_words(&maps.w[i], m.W, (uint64_t)m.rows, (uint64_t)p.NB * fmt_bytes(m.fmt), (uint64_t)m.pitch, (uint32_t)raw_pitch(m.fmt))) return false;
        p.tma |= 1 << i;
    }
    const size_t smem = p.stages * (size_t)p.b_stage + (size_t)p.raw_depth * slot + 1024;
#define NT_BLOCKS(M) case M: launch_blocks<M>(maps, p, parts, few, grid, smem, s); break
    switch (mask) {
        NT_BLOCKS(1); NT_BLOCKS(2); NT_BLOCKS(4); NT_BLOCKS(5); NT_BLOCKS(8); NT_BLOCKS(16);
        default: launch_blocks<31>(maps, p, parts, few, grid, smem, s); break;
    }
#undef NT_BLOCKS
    return true;
}

// The same over F32 tokens, or (x null) over tokens that split_activations laid out; what it needs beside them is memory of this call, at most what a device keeps between
// calls: long runs of tokens go through it in portions
bool gemm_blocks(const GemvMat* mats, int n_mat, int K, const float* x, const float* norm_w, float eps, const void* split, bool fine, int T, bool add, cudaStream_t s) {
    if (T <= 0 || !gemm_blocks_supported(mats, n_mat, K) || (reinterpret_cast<uintptr_t>(x) & 15)) return false;
    fine = fine && x;
    bool as_it_lies = !x;
    for (int i = 0; i < n_mat; i++) as_it_lies = as_it_lies && !has_mins(gemv_kq_format(mats[i].dtype));
    auto up256 = [](size_t n) { return (n + 255) / 256 * 256; };
    if (as_it_lies) {
        const size_t front = up256(plain_tokens_bytes(T));
        CallMemory memory(front + block_scratch_bytes(T), s);
        if (!memory.p) return false;
        return gemm_blocks(mats, n_mat, K, plain_tokens(memory.p, split, T, s), static_cast<uint8_t*>(memory.p) + front, T, add, s);
    }
    auto front_of = [&](int tokens) { return up256(block_tokens_bytes(tokens, K, fine)); };
    int portion = (T + 127) / 128 * 128;
    for (int n = 2; portion > 128 && front_of(portion) + block_scratch_bytes(portion) > CALL_MEMORY_KEPT; n++) portion = ((T + n - 1) / n + 127) / 128 * 128;
    portion = std::min(portion, T);
    CallMemory memory(front_of(portion) + block_scratch_bytes(portion), s);
    if (!memory.p) return false;
    const __half *hi = static_cast<const __half*>(split), *lo = hi + padded(T) * (size_t)K;
    GemvMat m[3];
    for (int t0 = 0; t0 < T; t0 += portion) {
        const int n = std::min(portion, T - t0);
        const size_t at = (size_t)t0 * K;
        for (int i = 0; i < n_mat; i++) { m[i] = mats[i]; m[i].y += (size_t)t0 * mats[i].out; }
        const BlockTokens t = x ? split_tokens(memory.p, x + at, norm_w, eps, n, K, fine, s) : resplit_tokens(memory.p, hi + at, lo + at, n, K, s);
        if (!gemm_blocks(m, n_mat, K, t, static_cast<uint8_t*>(memory.p) + front_of(portion), n, add, s)) return false;
    }
    return true;
}

void silu_mul_split(void* workspace, const float* gate, const float* up, int rows, int cols, cudaStream_t s) {
    const size_t Mp = ((size_t)rows + 127) / 128 * 128, n4 = (size_t)rows * cols / 4;
    __half* hi = static_cast<__half*>(workspace);
    silu_split_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, s>>>(reinterpret_cast<uint2*>(hi), reinterpret_cast<uint2*>(hi + Mp * (size_t)cols),
                                                                 reinterpret_cast<const float4*>(gate), reinterpret_cast<const float4*>(up), n4);
    count_launch();
}

}}  // namespace nt::b200
