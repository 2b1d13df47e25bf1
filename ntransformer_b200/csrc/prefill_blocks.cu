// prefill_blocks.cu — tensor-core GEMM of prompts over matrices in GGUF blocks: Y[T, N] (+)= X[T, K] . W[N, K]^T, W expanded on the way to the MMA.
//
// The reference has no batched product (prefill loops its GEMV over the tokens, src/model/attention.cpp:144-162, ffn.cpp:96-133).  The form this
// replaces wrote each matrix out as a pair of F16 matrices W_hi + W_lo (12 bytes of traffic for a 0.6-byte weight) and ran two GEMMs over it, four
// products of halves in all, on 128 x 256 tiles of which a narrow matrix fills few.  Here a CTA owns 128 rows of W and NT tokens:
//   * the roles of the operands are exchanged: W is A (M = 128 rows), tokens are B (N = NT, any multiple of 16 up to 256, chosen so that the tiles
//     fill whole waves of the SMs);
//   * sixteen warps expand 64 columns of the 128 rows at a time (eight each of two k-blocks in turn), a row to a lane: blocks come into shared memory by cp.async, the F32 value of a weight is
//     split into F16 hi + lo (W = hi + lo to 2^-22 of it, or to 2^-25 where that is more: the least F16 halved) and stored to TENSOR MEMORY, from where tcgen05.mma takes its A operand: shared memory's bandwidth
//     is left to B;
//   * B is the split of the tokens (prefill_gemm.cu's workspace) by TMA; three products hi.hi, hi.lo, lo.hi (lo.lo, up to 2^-22 of a product and of either
//     sign, leaves 4e-8 of a result; what follows is a hundred times that);
//   * half of K, at most 2048 columns, to an accumulator, partial sums added in F32 by the epilogue: the tensor cores cut off each addition, which leaves
//     1.86e-8 of the result for each.  The expanded form made 2 of them for 16 columns of up to 4096, this one makes 3 for 16 of half as many: error against 64 bits
//     2.5e-6 -> 2.0e-6 at K = 1024, 9.7e-6 -> 7.1e-6 at 4096 (whole rows to 2048 left 3.6e-6 at 1024).
// Llama-3 8B layer in Q4_K_M, 500 tokens: q/k/v 78 us (was 332 with the expansion), o 63 (173), gate + up 336 (604 and 40 for SwiGLU), down 201 (494); of
// 1.9 us per 64 columns at first, 0.9 went into an epilogue that read C back before each addition (now red.add), 0.2 into an MMA loop of one lane.
#include "kernels_internal.h"
#include "ring.cuh"
#include "tc_device.cuh"
#include "gemv_mma_device.cuh"
#include <algorithm>

namespace nt { namespace b200 {

namespace {

constexpr int QBK = 64;                                  // columns of a k-block: a 128-byte swizzle row of F16
constexpr int A_STAGES = 4, A_COLS = 64;             // tensor-memory columns of an expanded k-block: 32 hi, 32 lo; the accumulators lie behind them
constexpr int D_COL = A_STAGES * A_COLS;
constexpr int KC_MAX = 2048 / QBK;                       // k-blocks to an accumulator, at most
constexpr int B_STAGES_MAX = 4;
constexpr int Q_THREADS = 22 * 32;                       // warp 0 TMA, 1 MMA, 2-5 epilogue, 6-21 expansion

__host__ __device__ constexpr int raw_pitch(int fmt) { return fmt == 2 ? 240 : fmt_bytes(fmt); }       // odd 16-byte units; Q6_K: the 14 units around a block

struct BlkMat { const uint8_t* W; float* C; int rows, tiles, fmt; long long pitch; };
struct BlkParams {
    BlkMat mat[3];
    int n_mat, T, NT, cols, n_tiles, Mp, K, kc, add, b_stages, raw_depth, raw_slot, d_bufs;
    unsigned* status;          // wait_status.cuh
};

// tcgen05.mma with A in tensor memory
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const uint8_t* src, int bytes) {       // the first `bytes`, zeros behind them
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// 8 rows of super-block b into a slot: four lanes to a row, 64 contiguous bytes an instruction; rows behind the matrix are its last one, and nothing
// behind the matrix's end is read
template <int FMT>
__device__ __forceinline__ void copy_rows(uint32_t slot, const BlkMat& m, int row, int b, int NB, int lane) {
    constexpr int PITCH = raw_pitch(FMT), UNITS = FMT == 2 ? 14 : fmt_bytes(FMT) / 16;
    const uint8_t* end = m.W + (long long)(m.rows - 1) * m.pitch + (long long)NB * fmt_bytes(FMT);
    {
        const int r = lane >> 2;
        const uint8_t* p = m.W + (long long)min(row + r, m.rows - 1) * m.pitch + (long long)b * fmt_bytes(FMT);
        if (FMT == 2) p = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)15);
#pragma unroll
        for (int i = 0; i < (UNITS + 3) / 4; i++) {
            const int u = 4 * i + (lane & 3);
            if (u >= UNITS) break;
            const long long left = end - (p + 16 * u);
            copy16(slot + r * PITCH + 16 * u, left > 0 ? p + 16 * u : m.W, FMT == 2 ? (int)max(0ll, min(16ll, left)) : 16);
        }
    }
}

__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
// 32 consecutive weights of this lane's row — half hf of k-block c (0..3) of the super-block — as F16 pairs hi and lo, two columns of K to a word.
// blk: the block in shared memory.
template <int FMT>
__device__ __forceinline__ void expand32(const uint8_t* blk, int c, int hf, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
    uint32_t q[8];                                                 // codes, four to a word, unsigned
    float off, D[2], M;                                            // weight = D (code - off) - M, D of the first and the second 16
    M = 0.f;
    if (FMT <= 1) {
        const uint4 h = lds128(blk), a = lds128(blk + (FMT == 0 ? 16 : 48) + 32 * c), b = lds128(blk + (FMT == 0 ? 32 : 64) + 32 * c);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const int sub = 2 * c + hf;
        const uint32_t ss = sub < 4 ? h.y & 0x3F3F3F3Fu : (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
        const uint32_t mm = sub < 4 ? h.z & 0x3F3F3F3Fu : ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
        D[0] = D[1] = half_bits(h.x & 0xFFFFu) * magic_byte(ss, 0x7440u + (sub & 3));
        M = half_bits(h.x >> 16) * magic_byte(mm, 0x7440u + (sub & 3));
        off = 8388608.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = (w[i] >> (4 * hf)) & 0x0F0F0F0Fu;
        if (FMT == 1) {
            const uint4 e = lds128(blk + 16), f = lds128(blk + 32);
            const uint32_t v[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] |= ((v[i] >> sub) & 0x01010101u) << 4;
        }
    } else {
        auto words = [&](const uint8_t* p, uint32_t (&w)[8]) {     // 32 bytes from any even address
            const uint32_t mis = smem_u32(p) & 2u, sel = mis ? 0x5432u : 0x3210u;
            const uint32_t* a = reinterpret_cast<const uint32_t*>(p - mis);
            uint32_t u = a[0];
#pragma unroll
            for (int i = 0; i < 8; i++) { const uint32_t n = (i < 7 || mis) ? a[i + 1] : 0u; w[i] = __byte_perm(u, n, sel); u = n; }
        };
        if (FMT == 2) {
            // half h of the super-block, quarters q1 (codes in the low nibbles of the first 32 bytes, bits 0-1 of the pairs), q2 (second 32, bits 2-3), q3, q4
            const int h = c >> 1, qt = 2 * (c & 1) + hf;
            uint32_t w[8], v[8];
            words(blk + 64 * h + 32 * hf, w);
            words(blk + 128 + 32 * h, v);
            const float d = half_bits(*reinterpret_cast<const uint16_t*>(blk + 208));
            const int8_t* sc = reinterpret_cast<const int8_t*>(blk + 192 + 8 * h + 2 * qt);
            D[0] = d * (float)sc[0]; D[1] = d * (float)sc[1];
            off = 8388608.0f + 32.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] = ((w[i] >> (4 * (c & 1))) & 0x0F0F0F0Fu) | (((v[i] >> (2 * qt)) & 0x03030303u) << 4);
        } else if (FMT == 3) {
            const uint8_t* b = blk + 34 * (2 * c + hf);
            words(b + 2, q);
            D[0] = D[1] = half_bits(*reinterpret_cast<const uint16_t*>(b));
            off = 8388608.0f + 128.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] ^= 0x80808080u;
        } else {
            const uint8_t* b = blk + 18 * (2 * c + hf);
            const uint32_t mis = smem_u32(b + 2) & 2u, sel = mis ? 0x5432u : 0x3210u;
            const uint32_t* a = reinterpret_cast<const uint32_t*>(b + 2 - mis);
            D[0] = D[1] = half_bits(*reinterpret_cast<const uint16_t*>(b));
            off = 8388608.0f + 8.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t n = __byte_perm(a[i], (i < 3 || mis) ? a[i + 1] : 0u, sel);
                q[i] = n & 0x0F0F0F0Fu;
                q[4 + i] = (n >> 4) & 0x0F0F0F0Fu;
            }
        }
    }
    const uint64_t off2 = pack2(-off, -off), m2 = pack2(-M, -M), one2 = pack2(-1.0f, -1.0f);
#pragma unroll
    for (int i = 0; i < 16; i++) {                                 // two weights at a time in packed F32 arithmetic
        const float d = D[i >> 3];
        const uint32_t w4 = q[i >> 1];
        uint64_t w = add2(pack2(__uint_as_float(__byte_perm(w4, 0x4B000000u, 0x7440u + 2 * (i & 1))), __uint_as_float(__byte_perm(w4, 0x4B000000u, 0x7441u + 2 * (i & 1)))), off2);
        w = fma2(w, pack2(d, d), m2);
        float a, b;
        unpack2(w, a, b);
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        unpack2(fma2(pack2(f.x, f.y), one2, w), a, b);             // w - hi, exact
        const __half2 l = __floats2half2_rn(a, b);
        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
        lo[i] = *reinterpret_cast<const uint32_t*>(&l);
    }
}

__global__ void __launch_bounds__(Q_THREADS, 1) gemm_blocks_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ BlkParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t b_full[B_STAGES_MAX], b_empty[B_STAGES_MAX], a_full[A_STAGES], a_empty[A_STAGES], d_full[2], d_empty[2];
    __shared__ uint32_t tmem_base_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NB = p.K / 256, num_kb = p.K / QBK, n_kc = (num_kb + p.kc - 1) / p.kc, NT = p.NT;
    const uint32_t b_tile = (uint32_t)NT * 128, b_stage = 2 * b_tile;
    uint8_t* raw = smem + (size_t)p.b_stages * b_stage;
    auto place = [&](int tile, int& mi, int& row0, int& t0) {      // tokens inside: the CTAs of a wave share rows
        const int rt = tile / p.cols;
        t0 = (tile - rt * p.cols) * NT;
        mi = 0;
        int r = rt;
        while (mi + 1 < p.n_mat && r >= p.mat[mi].tiles) { r -= p.mat[mi].tiles; mi++; }
        row0 = r * 128;
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.b_stages; i++) { mbar_init(b_full + i, 1); mbar_init(b_empty + i, 1); }
        for (int i = 0; i < A_STAGES; i++) { mbar_init(a_full + i, 8); mbar_init(a_empty + i, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(d_full + i, 1); mbar_init(d_empty + i, 4); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_smem;

    if (warp == 0) {
        if (lane == 0) {                                           // ---- tokens by TMA ----
            uint32_t st = 0, par = 1, filled = 0;
            uint32_t tries = WAIT_TRIES;                                     // 0: a wait of this thread has run out
            for (int tile = blockIdx.x; tile < p.n_tiles && tries; tile += gridDim.x) {
                int mi, row0, t0;
                place(tile, mi, row0, t0);
                for (int kb = 0; kb < num_kb; kb++) {
                    wait_phase(b_empty + st, par, p.status, tries);
                    if (!tries) {
                        for (uint32_t s = 0; s < filled; s++) wait_flight(b_full + s, s < st ? par ^ 1u : par);      // the copies in flight
                        break;
                    }
                    filled = min(filled + 1, (uint32_t)p.b_stages);
                    uint8_t* d = smem + (size_t)st * b_stage;
                    mbar_expect_tx(b_full + st, b_stage);
                    tma_load_2d(d, &map_x, kb * QBK, t0, b_full + st);
                    tma_load_2d(d + b_tile, &map_x, kb * QBK, p.Mp + t0, b_full + st);      // the lo halves lie Mp rows below
                    if (++st == (uint32_t)p.b_stages) { st = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA: the whole warp walks the loop, so that addresses and descriptors stay in uniform registers, and one lane issues (a loop of lane 0
        // alone moved every operand of every MMA there: about 100 cycles an instruction) ----
        const bool leader = elect_lane();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | (8u << 24);      // D F32, A and B F16 K-major, N, M = 128
        const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem, 0);
        const uint64_t desc0 = make_desc(smem), lo_step = (uint64_t)(b_tile >> 4), stage_step = (uint64_t)(b_stage >> 4);
        uint32_t bs = 0, bpar = 0, as = 0, apar = 0, db = 0, dpar = 1;
        uint32_t tries = WAIT_TRIES;                                         // 0: a wait of this lane has run out
        int last = -1;                                             // stage and parity of the last commit
        for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x)
            for (int kc = 0; kc < n_kc; kc++) {
                wait_phase(d_empty + db, dpar, p.status, tries);
                const uint32_t d = tm + D_COL + db * NT;
                const int kb0 = kc * p.kc, kb1 = min(num_kb, kb0 + p.kc);
                for (int kb = kb0; kb < kb1; kb++) {
                    wait_phase(b_full + bs, bpar, p.status, tries);
                    wait_phase(a_full + as, apar, p.status, tries);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bh = desc0 + bs * stage_step, bl = bh + lo_step;
                    const uint32_t ah = tm + as * A_COLS, al = ah + 32;
                    if (leader && tries) {
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ts(d, al + 8 * k, bh + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);      // the small products first
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ts(d, ah + 8 * k, bl + 2 * k, idesc, 1u);
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ts(d, ah + 8 * k, bh + 2 * k, idesc, 1u);
                        umma_commit(b_empty + bs);
                        umma_commit(a_empty + as);
                        last = (int)(as * 2 + apar);
                        if (kb + 1 == kb1) umma_commit(d_full + db);
                    }
                    __syncwarp();
                    if (++bs == (uint32_t)p.b_stages) { bs = 0; bpar ^= 1; }
                    if (++as == A_STAGES) { as = 0; apar ^= 1; }
                }
                if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
            }
        if (!tries && last >= 0) wait_flight(a_empty + (last >> 1), last & 1);      // given up: the products in flight
    } else if (warp < 6) {                                         // ---- epilogue: a lane is a row of W, so a warp stores 128 contiguous bytes for each token ----
        const int quarter = warp & 3;
        uint32_t db = 0, dpar = 0;
        uint32_t tries = WAIT_TRIES;
        for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
            int mi, row0, t0;
            place(tile, mi, row0, t0);
            const BlkMat& m = p.mat[mi];
            const int row = row0 + quarter * 32 + lane, live = min(NT, p.T - t0);
            for (int kc = 0; kc < n_kc; kc++) {
                wait_phase(d_full + db, dpar, p.status, tries);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + D_COL + db * NT;
                const bool add = p.add || kc > 0;
                float* c = m.C + (size_t)t0 * m.rows + row;
#pragma unroll 1
                for (int n = 0; n < live; n += 32) {               // an odd multiple of 16: the last 16 columns read are not this tile's (nor beyond the 512), and not used
                    uint32_t v[32];
                    tmem_ld32(d + (uint32_t)n, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (row < m.rows && tries) {
                        // adds go to the memory's side (this lane is the element's only writer, so their order is fixed): nothing is waited for
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            if (n + j >= live) break;
                            float* o = c + (size_t)(n + j) * m.rows;
                            if (add) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(o), "f"(__uint_as_float(v[j])) : "memory");
                            else *o = __uint_as_float(v[j]);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0 && tries) mbar_arrive(d_empty + db);
                if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
            }
        }
    } else {                                                       // ---- expansion: four warps share 32 rows; half hf of the k-blocks 0, 2 or 1, 3 of a super-block to each ----
        const int quarter = warp & 3, share = (warp - 6) >> 2, hf = share & 1, odd = share >> 1, depth = p.raw_depth;
        uint8_t* ring = raw + (size_t)quarter * depth * p.raw_slot;
        uint32_t as = odd, apar = 1;
        // the sequence of super-blocks over this CTA's tiles, `depth - 1` copied ahead
        int ct = blockIdx.x, cb = 0, cslot = 0, cmi = 0, crow = 0, ct0 = 0;
        if (ct < p.n_tiles) place(ct, cmi, crow, ct0);
        auto copy_next = [&]() {
            if (ct < p.n_tiles) {
                const BlkMat& m = p.mat[cmi];
                const uint32_t dst = smem_u32(ring + (size_t)cslot * p.raw_slot) + (uint32_t)(share * 8 * raw_pitch(m.fmt));
                const int row = crow + quarter * 32 + share * 8;
                switch (m.fmt) {
                    case 0: copy_rows<0>(dst, m, row, cb, NB, lane); break;
                    case 1: copy_rows<1>(dst, m, row, cb, NB, lane); break;
                    case 2: copy_rows<2>(dst, m, row, cb, NB, lane); break;
                    case 3: copy_rows<3>(dst, m, row, cb, NB, lane); break;
                    default: copy_rows<4>(dst, m, row, cb, NB, lane); break;
                }
                if (++cb == NB) { cb = 0; ct += gridDim.x; if (ct < p.n_tiles) place(ct, cmi, crow, ct0); }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (++cslot == depth) cslot = 0;
        };
        for (int i = 0; i < depth - 1; i++) copy_next();
        int slot = 0, pending = -1;
        uint32_t tries = WAIT_TRIES;
        auto stored = [&](int stage) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0 && tries) mbar_arrive(a_full + stage);
        };
        for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
            int mi, row0, t0;
            place(tile, mi, row0, t0);
            const BlkMat& m = p.mat[mi];
            const int fmt = m.fmt, row = min(row0 + quarter * 32 + lane, m.rows - 1);
            for (int b = 0; b < NB; b++) {
                if (depth == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                named_sync<128>(1 + quarter);                      // all rows have arrived, and all four warps are done with the slot copied into next
                copy_next();
                const uint8_t* blk = ring + (size_t)slot * p.raw_slot + lane * raw_pitch(fmt);
                if (fmt == 2) blk += (int)(((uint64_t)row * (uint64_t)m.pitch + (uint64_t)b * 210u) & 15u);
                if (++slot == depth) slot = 0;
#pragma unroll 1
                for (int c = odd; c < 4; c += 2) {
                    uint32_t hi[16], lo[16];
                    switch (fmt) {
                        case 0: expand32<0>(blk, c, hf, hi, lo); break;
                        case 1: expand32<1>(blk, c, hf, hi, lo); break;
                        case 2: expand32<2>(blk, c, hf, hi, lo); break;
                        case 3: expand32<3>(blk, c, hf, hi, lo); break;
                        default: expand32<4>(blk, c, hf, hi, lo); break;
                    }
                    // the stores of the k-block before had this one's arithmetic to arrive in
                    if (pending >= 0) stored(pending);
                    wait_phase(a_empty + as, apar, p.status, tries);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a = tmem + ((uint32_t)(quarter * 32) << 16) + as * A_COLS + hf * 16;
                    tmem_st16(a, hi);
                    tmem_st16(a + 32, lo);
                    pending = (int)as;
                    as += 2;
                    if (as >= A_STAGES) { as = odd; apar ^= 1; }
                }
            }
        }
        if (pending >= 0) stored(pending);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
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

}  // namespace

bool gemm_blocks_supported(const GemvMat* mats, int n_mat, int K) { return gemv_kq_any_pitch(mats, n_mat, K); }

// C_i [T, rows_i] (+)= X . W_i^T with X split into `workspace` (split_activations / rmsnorm_split: hi rows, then lo rows Mp below)
bool gemm_blocks(const GemvMat* mats, int n_mat, int K, const void* workspace, int T, bool add, cudaStream_t s) {
    if (T <= 0 || !gemm_blocks_supported(mats, n_mat, K)) return false;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    BlkParams p{};
    p.status = wait_status();
    p.n_mat = n_mat; p.T = T; p.K = K; p.add = add;
    p.kc = std::min(KC_MAX, (K / QBK + 1) / 2);
    p.Mp = (T + 127) / 128 * 128;
    int tiles = 0, slot = 0;
    for (int i = 0; i < n_mat; i++) {
        BlkMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W); m.C = mats[i].y; m.rows = mats[i].out; m.tiles = (m.rows + 127) / 128;
        m.fmt = gemv_kq_format(mats[i].dtype);
        m.pitch = (long long)(mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K));
        tiles += m.tiles;
        if (32 * raw_pitch(m.fmt) > slot) slot = 32 * raw_pitch(m.fmt);
    }
    // Tokens of a tile: the split of T that costs least in waves of the SMs times a tile's cycles for 64 columns, measured as 1050 + 5.7 NT (0.79, 0.98, 1.1
    // and 1.3 us at 64, 128, 176 and 256 tokens: the expansion's instructions up to about 100 tokens, then MMA and the tokens' loads).
    long long best = -1;
    for (int cols = (T + 255) / 256; cols <= (T + 31) / 32; cols++) {
        const int NT = ((T + cols - 1) / cols + 15) / 16 * 16, n = (T + NT - 1) / NT;
        const long long cost = ((long long)tiles * n + sms - 1) / sms * (10500 + 57 * NT);
        if (best < 0 || cost < best) { best = cost; p.NT = NT; p.cols = n; }
    }
    p.n_tiles = tiles * p.cols;
    p.d_bufs = 2 * p.NT <= 512 - A_STAGES * A_COLS ? 2 : 1;
    p.raw_slot = slot;
    const size_t cap = 226 * 1024 - 1024, b_stage = (size_t)p.NT * 256;
    p.raw_depth = 2 * b_stage + 4 * 3 * (size_t)slot <= cap ? 3 : 2;
    p.b_stages = (int)((cap - 4 * (size_t)p.raw_depth * slot) / b_stage);
    if (p.b_stages > B_STAGES_MAX) p.b_stages = B_STAGES_MAX;
    if (p.b_stages < 1) return false;
    CUtensorMap map;
    if (!tc_map_f16(&map, workspace, 2 * (uint64_t)p.Mp, (uint64_t)K, (uint32_t)p.NT)) return false;
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(gemm_blocks_kernel, 226 * 1024, configured);
    gemm_blocks_kernel<<<p.n_tiles < sms ? p.n_tiles : sms, Q_THREADS, p.b_stages * b_stage + 4 * (size_t)p.raw_depth * slot + 1024, s>>>(map, p);
    count_launch();
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
