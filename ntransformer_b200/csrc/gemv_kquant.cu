// gemv_kquant.cu — dequant-fused GEMV over GGUF Q4_K / Q5_K / Q6_K / Q8_0 / Q4_0 blocks for sm_100a.
//
// Replaces reference kernels K1-K5 (src/cuda/gemm.cu:32-470) behind launch_gemv (gemm.cu:748-805), and RMSNorm (rmsnorm.cu:17-70) in front of it.
// Bound by HBM for the large matrices and by launch and latency for the small ones, so:
//   * the products run on matrix instructions (gemv_mma_device.cuh);
//   * a team of KW warps takes 16 rows at a time and shares K, one or two super-blocks of every stage each.  A producer warp streams the rows through
//     the team's ring of stages (a cp.async.bulk for each row, mbarriers).  At the end of the rows the warps' shares meet in shared memory in a fixed
//     order (deterministic);
//   * several teams on an SM, so that the barriers of one do not idle it.  Weights depend on no kernel in flight: under programmatic launch a
//     kernel's first stages are fetched while the one before still runs, as far as it leaves room.  The activation vector is read after
//     griddepcontrol.wait, and the dependants are released after it;
//   * the prologue quantises the F32 vector (24-bit integers for each 32-block, 32-bit ones on request in front of Q4_0) into shared memory, with RMSNorm's
//     gains multiplied in and its scalar applied to the results.
// Up to 3 matrices of mixed formats share a launch (q / k / v of a Q4_K_M file; gate + up with SwiGLU).
#include "kernels_internal.h"
#include "ring.cuh"
#include "xquant.cuh"
#include "gemv_mma_device.cuh"
#include <cuda_fp16.h>
#include <algorithm>
#include <cstdlib>

namespace nt { namespace b200 {

namespace {

constexpr int MAX_MATS = 3;
constexpr int MAX_K = 49152;
constexpr int MAX_STAGES = 8;
constexpr int MAX_TEAMS = 4;
constexpr int SM_WARPS = 16;           // warps that multiply on an SM: TEAMS * KW in each of SM_WARPS / (TEAMS * KW) CTAs

struct KqMat {
    const uint8_t* W;
    float* y;
    int out;
    int groups;        // ceil(out / 16)
    int fmt;           // 0 Q4_K, 1 Q5_K, 2 Q6_K, 3 Q8_0 (as groups of 8 blocks), 4 Q4_0 (likewise)
    long long row_pitch;
};
struct KqParams {
    KqMat mat[MAX_MATS];
    int n_mat;
    int K, NB;                 // elements, super-blocks per row
    const int8_t* xq;          // pre-quantised activations (kernels_internal.h "xq"), or null:
    const float* x_f32;        //   F32 activations quantised in the prologue,
    const float* norm_w;       //   optionally as RMSNorm(x) * norm_w: the prologue quantises x * norm_w and sums x^2 in the same
    float eps;                 //   pass; the scalar rsqrt(mean(x^2) + eps) is applied to the results (exact up to round-off)
    int total_groups;          // groups of 16 rows of a matrix; SWIGLU: pairs of them, gate and up (two segments), or 8 rows of gate and the same 8 of up (halves)
    int n_seg;                 // segments (matrices) per group
    int halves;
    int weights_settled;       // no launch still under way writes the weights: they are read ahead of the wait for the launch before
    int epilogue;
    int stages, slot;          // depth of a team's ring and bytes of a stage
    unsigned* status;          // wait_status.cuh
    PeerOut peer;              // epilogue GEMV_PEER
};

// Shared memory: [barriers][zeros][norm][a wait has run out][partials][digit planes][scales(, those of the upper digits)][sums][rings]
constexpr size_t SM_ZERO = MAX_TEAMS * 16 * MAX_STAGES, SM_RED = SM_ZERO + 16, SM_DEAD = SM_RED + 64, SM_PART = SM_RED + 112;
constexpr size_t SM_X = (SM_PART + SM_WARPS * 2 * 2 * MROWS * 4 + 127) & ~(size_t)127;
__host__ __device__ constexpr size_t x_bytes(int K, int planes) { return ((size_t)planes * (K + 64) + (size_t)(K / 32) * (planes == 4 ? 12 : 8) + 127) & ~(size_t)127; }
// Kernels whose vector may have four digits (GemvInput::whole, where there is room): launch_gemv multiplied Q4_0 in F32, and three digits left more error than that
// (4096 wide, one element in a hundred ten times the others: 1.6e-7 of the result, 1.2e-7 in F32 and 1.0e-7 with four).  The digit's column of the product was
// zeros, but the prologue and the vector's place in shared memory grow: decode step of four 8B layers in Q4_0 309 us with four, 302 with three.
constexpr int WHOLE = 32;               // in a kernel's MASK, beside the format's bit

// Eight consecutive elements (t8 = their index / 8), four threads to a 32-element block: digits, scale and sum into shared memory.
template <int MASK>
__device__ __forceinline__ void quantize8(const float (&x)[8], int t8, uint8_t* planes, int plane, float* xs, float* xs_upper, float* sums) {
    constexpr bool FOUR = MASK & WHOLE;
    float amax = 0.f, s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) { amax = fmaxf(amax, fabsf(x[i])); s = __fadd_rn(s, x[i]); }
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, 1));
    s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, 2));
    constexpr float top = FOUR ? BlockScale::TOP4 : BlockScale::TOP3;
    const BlockScale scale(amax, top);
    uint32_t d[4][2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int T[4];
        scale.integers<(MASK & (4 | 16)) != 0>(x + 4 * h, T);
        if (FOUR) digits4(T, d[0][h], d[1][h], d[2][h], d[3][h]);
        else { digits4(T, d[0][h], d[1][h], d[2][h]); d[3][h] = 0; }
    }
    const uint32_t o = xword_byte(t8 * 8);                      // the two words are neighbours in t: 16 bytes apart
#pragma unroll
    for (int p = 0; p < (FOUR ? 4 : 3); p++) {
        *reinterpret_cast<uint32_t*>(planes + p * plane + o) = d[p][0];
        *reinterpret_cast<uint32_t*>(planes + p * plane + o + 16) = d[p][1];
    }
    if ((t8 & 3) == 0) {
        const int b = t8 >> 2;                                  // 32-element block: 2 c + hi of its super-block
        const float f = BlockScale::of(amax, s, top);
        xs[(b & ~7) + (b & 1) * 4 + ((b & 7) >> 1)] = f;
        if (FOUR) xs_upper[(b & ~7) + (b & 1) * 4 + ((b & 7) >> 1)] = f * 65536.0f;
        sums[b] = s;
    }
}

// MASK: bit f set <=> matrices of format f may appear in this launch (mixed Q4_K_M projections share one launch).
template <int MASK, int KW, int TEAMS>
__global__ void __launch_bounds__(TEAMS * (KW + 1) * 32, SM_WARPS / (TEAMS * KW)) gemv_mma_kernel(const __grid_constant__ KqParams p) {
    constexpr int CTHREADS = TEAMS * KW * 32, np = MASK & WHOLE ? 4 : 3;      // np: digits of an activation
    extern __shared__ __align__(128) uint8_t smem[];
    const int team = (int)threadIdx.x / ((KW + 1) * 32);
    const int warp = (threadIdx.x >> 5) - team * (KW + 1), lane = threadIdx.x & 31;
    const int stages = p.stages, slot_bytes = p.slot;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem) + team * 2 * MAX_STAGES;
    uint64_t* empty = full + MAX_STAGES;
    uint8_t* ring = smem + SM_X + x_bytes(p.K, np) + (size_t)team * stages * slot_bytes;
    const int u0 = (int)blockIdx.x + team * (int)gridDim.x, ustep = (int)gridDim.x * TEAMS;      // few groups: a team in each CTA first
    auto format = [&](const KqMat& m) { return (MASK == 1) ? 0 : (MASK == 2) ? 1 : (MASK == 4) ? 2 : (MASK == 8) ? 3 : (MASK & 16) ? 4 : m.fmt; };
    auto locate = [&](int u, int seg, int& mi, int& gl) {       // matrix and local group of group u
        if (p.n_seg == 2 || p.halves) { mi = seg; gl = u; return; }
        mi = 0; gl = u;
        while (mi + 1 < p.n_mat && gl >= p.mat[mi].groups) { gl -= p.mat[mi].groups; mi++; }
    };
    if (warp == KW && lane == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(full + s, 1); mbar_init(empty + s, KW); }
        mbar_fence_init();
    }
    if (threadIdx.x < 4) reinterpret_cast<uint32_t*>(smem + SM_ZERO)[threadIdx.x] = 0;
    const uint32_t dead = smem_u32(smem + SM_DEAD);
    if (threadIdx.x == 4) set_word(dead, 0u);
    __syncthreads();

    if (warp == KW) {                                           // ---- producer: lane r < 16 copies row r of each stage ----
        int slot = 0;
        uint32_t parity = 1;                                    // the first round finds every slot empty
        bool ahead = true;                                      // still in it
        if (!p.weights_settled) pdl_wait();
        for (int u = u0; u < p.total_groups; u += ustep) {
            for (int seg = 0; seg < p.n_seg; seg++) {
                int mi, gl;
                locate(u, seg, mi, gl);
                if (p.halves) mi = (lane >> 3) & 1;
                const KqMat& m = p.mat[mi];
                const int fmt = format(p.mat[p.halves ? 0 : mi]), blk = fmt_bytes(fmt), sblocks = stage_blocks(fmt, KW), row = p.halves ? gl * 8 + (lane & 7) : gl * MROWS + lane;
                const uint8_t* end = m.W + (long long)(m.out - 1) * m.row_pitch + (long long)p.NB * blk;       // of the matrix
                for (int b0 = 0; b0 < p.NB; b0 += sblocks) {
                    // whole 16-byte units around the row's bytes; what of the last one lies behind the matrix is left out and copied singly
                    const uint8_t* b = m.W + (long long)row * m.row_pitch + (long long)b0 * blk;
                    const uint8_t* b16 = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(b) & ~(uintptr_t)15);
                    const uint8_t* e = b + min(sblocks, p.NB - b0) * blk;
                    const uint8_t* e16 = reinterpret_cast<const uint8_t*>((reinterpret_cast<uintptr_t>(e) + 15) & ~(uintptr_t)15);
                    if (e16 > end) e16 -= 16;
                    const uint32_t bytes = lane < MROWS && row < m.out ? (uint32_t)(e16 - b16) : 0u;
                    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, bytes);
                    if (!ahead) wait_cta(empty + slot, parity, dead);
                    uint8_t* dst = ring + (size_t)slot * slot_bytes + lane * stage_pitch(fmt, KW);
                    if (bytes && e16 < e)
                        for (const uint8_t* q = e16; q < e; q += 2) *reinterpret_cast<uint16_t*>(dst + (q - b16)) = *reinterpret_cast<const uint16_t*>(q);
                    __syncwarp();
                    if (lane == 0) mbar_expect_tx(full + slot, total);
                    __syncwarp();
                    if (bytes) bulk_g2s(dst, b16, bytes, full + slot);
                    if (++slot == stages) {
                        slot = 0; parity ^= 1u;
                        if (ahead) { pdl_wait(); ahead = false; }   // the readers start there too: from now on a wait is a short one
                    }
                }
            }
        }
        if (word_set(dead))                                     // given up: the copies in flight (parity counts for slots yet to be filled in this round)
            for (int s = 0; s < (ahead ? slot : stages); s++) wait_flight(full + s, s < slot ? parity ^ 1u : parity);
        return;
    }

    // ---- the activation vector into shared memory ----
    pdl_wait();
    pdl_launch_dependents();
    const int K = p.K, plane = K + 64, tid = team * KW * 32 + warp * 32 + lane;
    uint8_t* planes = smem + SM_X;
    float* xs = reinterpret_cast<float*>(planes + np * (size_t)plane);
    float* xs_upper = xs + K / 32;                              // four digits
    float* sums = np == 4 ? xs_upper + K / 32 : xs_upper;
    float* red = reinterpret_cast<float*>(smem + SM_RED);
    float rms_inv = 1.0f;
    if (p.x_f32) {
        const float *x_f32 = behind_wait(p.x_f32), *norm_w = behind_wait(p.norm_w);
        float ss = 0.f;
        constexpr int AHEAD = 4;                                // vectors of 8 in flight for each thread
        for (int base = 0; base < K / 8; base += AHEAD * CTHREADS) {
            float4 v[AHEAD][2];
#pragma unroll
            for (int j = 0; j < AHEAD; j++) {
                const int t8 = base + j * CTHREADS + tid;
                if (t8 < K / 8) { v[j][0] = __ldcg(reinterpret_cast<const float4*>(x_f32) + 2 * t8); v[j][1] = __ldcg(reinterpret_cast<const float4*>(x_f32) + 2 * t8 + 1); }
            }
#pragma unroll
            for (int j = 0; j < AHEAD; j++) {
                const int t8 = base + j * CTHREADS + tid;
                if (t8 >= K / 8) break;                         // K / 8 is a multiple of 32: whole warps leave together
                float x[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
                if (p.norm_w) {
                    const float4 a = __ldg(reinterpret_cast<const float4*>(norm_w) + 2 * t8), b = __ldg(reinterpret_cast<const float4*>(norm_w) + 2 * t8 + 1);
                    const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                    for (int i = 0; i < 8; i++) { ss = fmaf(x[i], x[i], ss); x[i] = __fmul_rn(x[i], w[i]); }
                }
                quantize8<MASK>(x, t8, planes, plane, xs, xs_upper, sums);
            }
        }
        if (p.norm_w) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
            if (lane == 0) red[team * KW + warp] = ss;
        }
    } else {
        // the public xq form: x = scale * (q1 * 16384 + q2 * 128 + q3), planes in 16-byte columns swizzled as xquant.cuh has it.  Times 4 the
        // integer splits into balanced bytes without a loss.
        const uint8_t* xq = reinterpret_cast<const uint8_t*>(behind_wait(p.xq));
        const float* fs = reinterpret_cast<const float*>(xq + 3 * (size_t)K);
        for (int e = 4 * tid; e < K; e += 4 * CTHREADS) {
            const uint32_t o = xq_swizzle((uint32_t)e);
            const uint32_t a = __ldg(reinterpret_cast<const uint32_t*>(xq + o)), b = __ldg(reinterpret_cast<const uint32_t*>(xq + K + o)),
                           c = __ldg(reinterpret_cast<const uint32_t*>(xq + 2 * (size_t)K + o));
            int T[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                T[i] = 4 * ((((int)(a << (24 - 8 * i)) >> 24) * 128 + ((int)(b << (24 - 8 * i)) >> 24)) * 128 + ((int)(c << (24 - 8 * i)) >> 24));
            uint32_t d[4] = {};
            if (np == 4) {
#pragma unroll
                for (int i = 0; i < 4; i++) T[i] *= 256;
                digits4(T, d[0], d[1], d[2], d[3]);
            } else digits4(T, d[0], d[1], d[2]);
#pragma unroll
            for (int q = 0; q < np; q++) *reinterpret_cast<uint32_t*>(planes + q * plane + xword_byte(e)) = d[q];
            if ((e & 31) == 0) {
                const int blk = e >> 5;
                const int at = (blk & ~7) + (blk & 1) * 4 + ((blk & 7) >> 1);
                xs[at] = (np == 4 ? 0.25f / 256.0f : 0.25f) * __ldg(fs + blk);
                if (np == 4) xs_upper[at] = 0.25f * 256.0f * __ldg(fs + blk);
                sums[blk] = __ldg(fs + K / 32 + 2 * blk) + __ldg(fs + K / 32 + 2 * blk + 1);
            }
        }
    }
    unsigned peer_seq = 0, peer_parity = 0;
    if (p.epilogue == GEMV_PEER) { peer_seq = __ldcg(p.peer.seq) + 1u; peer_parity = peer_seq & 1u; }
    named_sync<CTHREADS>(1);
    if (p.norm_w && p.x_f32) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < TEAMS * KW; i++) s += red[i];       // fixed order: the same value in every warp and CTA
        rms_inv = rsqrtf(s / K + p.eps);
    }
    const int g = lane >> 2, t = lane & 3;
    XView xv;
    const bool c0 = g < np, c1 = g >= 4 && g < 4 + np;
    xv.b0 = c0 ? planes + g * plane + t * 16 : smem + SM_ZERO;
    xv.b1 = c1 ? planes + (g - 4) * plane + t * 16 : smem + SM_ZERO;
    xv.m0 = c0 ? ~0u : 0u; xv.m1 = c1 ? ~0u : 0u;
    xv.xs = np == 4 && !(t & 1) ? xs_upper : xs; xv.sums = sums;

    float* part = reinterpret_cast<float*>(smem + SM_PART) + team * 2 * 2 * KW * MROWS;      // [buffer][segment][K share][row]
    int slot = 0, buf = 0, turn = 0;
    uint32_t parity = 0;
    for (int u = u0; u < p.total_groups; u += ustep) {
        for (int seg = 0; seg < p.n_seg; seg++) {
            int mi, gl;
            locate(u, seg, mi, gl);
            const KqMat& m = p.mat[mi];
            const int fmt = format(m), blk = fmt_bytes(fmt), sblocks = stage_blocks(fmt, KW);
            float acc[2] = {}, mins[2] = {};
            for (int b0 = 0; b0 < p.NB; b0 += sblocks) {
                const int sbi = b0 + warp, left = p.NB - sbi;   // super-blocks from this warp's first on
                wait_cta(full + slot, parity, dead);
                if (left > 0) {
                    const uint8_t* sb = ring + (size_t)slot * slot_bytes + warp * blk;
                    const bool two = KW == 4 && left > KW;
                    if ((MASK & 1) && fmt == 0) { if (two) tile_blocks<0, 2, KW>(sb, 0, sbi, xv, lane, acc, mins); else tile_blocks<0, 1, KW>(sb, 0, sbi, xv, lane, acc, mins); }
                    if ((MASK & 2) && fmt == 1) { if (two) tile_blocks<1, 2, KW>(sb, 0, sbi, xv, lane, acc, mins); else tile_blocks<1, 1, KW>(sb, 0, sbi, xv, lane, acc, mins); }
                    if ((MASK & 4) && fmt == 2)
                        tile_blocks<2, 1, KW>(sb, (int)((uint64_t)(gl * (p.halves ? 8 : MROWS) + g) * (uint64_t)m.row_pitch + (uint32_t)(b0 * 210) & 15u), sbi, xv, lane, acc, mins);
                    if ((MASK & 8) && fmt == 3) tile_blocks<3, 1, KW>(sb, 0, sbi, xv, lane, acc, mins);
                    if ((MASK & 16) && fmt == 4) { if (two) tile_blocks<4, 2, KW>(sb, 0, sbi, xv, lane, acc, mins); else tile_blocks<4, 1, KW>(sb, 0, sbi, xv, lane, acc, mins); }
                }
                __syncwarp();
                if (lane == 0) arrive(empty + slot);
                if (++slot == stages) { slot = 0; parity ^= 1u; }
            }
            const float f = lane_factor(fmt, t, np);
            // over the four lanes of a row pair: lane t = 0 ends with row g, t = 1 with row g + 8
            const float v0 = fmaf(acc[0], f, -mins[0]), v1 = fmaf(acc[1], f, -mins[1]);
            float v = (t & 1) ? v1 : v0;
            v += __shfl_xor_sync(0xFFFFFFFFu, (t & 1) ? v0 : v1, 1);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
            if (t < 2) part[((buf * 2 + seg) * KW + warp) * MROWS + g + 8 * t] = v;
        }
        named_sync<KW * 32>(2 + team);
        if (warp == turn && lane < MROWS) {                     // one warp in turn adds the shares and applies the epilogue
            const float* pw = part + buf * 2 * KW * MROWS + lane;
            float v0 = 0.f, v1 = 0.f;
#pragma unroll
            for (int w = 0; w < KW; w++) v0 += pw[w * MROWS];
            if (p.n_seg == 2) {
#pragma unroll
                for (int w = 0; w < KW; w++) v1 += pw[(KW + w) * MROWS];
            }
            const float other = __shfl_down_sync(0xFFFFu, v0, 8);
            if (p.halves) v1 = other;                           // up's row, eight lanes on
            v0 *= rms_inv; v1 *= rms_inv;                       // 1.0 unless the prologue normalised (RMSNorm's scalar factor)
            int mi, gl;
            locate(u, 0, mi, gl);
            const KqMat& m = p.mat[mi];
            const int row = p.halves ? gl * 8 + lane : gl * MROWS + lane;
            if (row < m.out && !(p.halves && lane >= 8)) {
                if (p.epilogue == GEMV_SWIGLU) {
                    // silu(g) * u with the reference's fast-math expression (gemm.cu:713-725)
                    m.y[row] = __fdividef(v0, 1.0f + __expf(-v0)) * v1;
                } else if (p.epilogue == GEMV_ADD) {
                    m.y[row] += v0;
                } else if (p.epilogue == GEMV_PEER) {
                    // this rank's partial row -> slot [parity][rank] on every rank: one 64-bit NVLink store {sequence : value} per peer
                    // (16 lanes write 128 contiguous bytes); the value is its own arrival flag
                    const size_t off = ((size_t)peer_parity * p.peer.size + p.peer.rank) * (size_t)p.peer.hidden + (size_t)row;
                    const unsigned long long pkt = ((unsigned long long)peer_seq << 32) | (unsigned long long)__float_as_uint(v0);
                    for (int r = 0; r < p.peer.size; r++)
                        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p.peer.slots[r] + off), "l"(pkt) : "memory");
                } else {
                    m.y[row] = v0;
                }
            }
        }
        buf ^= 1;
        if (++turn == KW) turn = 0;
    }
    if (word_set(dead)) {                                       // a wait ran out: no results
        report(p.status);
        for (int u = u0; u < p.total_groups && p.epilogue != GEMV_PEER; u += ustep) {
            int mi, gl;
            locate(u, 0, mi, gl);
            const int row = p.halves ? gl * 8 + lane : gl * MROWS + lane;
            if (lane < (p.halves ? 8 : MROWS) && row < p.mat[mi].out) p.mat[mi].y[row] = __uint_as_float(0x7FFFFFFFu);      // NaN
        }
    }
}

// Q4_0 (reference K1, gemm.cu:32-86) runs on this path by default; NT_B200_Q4_0_TMA=0 sends it back to the generic kernel (gemv_generic.cu) for
// A/B comparisons.
bool q4_0_tma_enabled() {
    static const bool on = [] { const char* e = getenv("NT_B200_Q4_0_TMA"); return !(e && e[0] == '0' && e[1] == 0); }();
    return on;
}
int fmt_of(DType dt) {
    return dt == DType::Q4_K_M ? 0 : dt == DType::Q5_K ? 1 : dt == DType::Q6_K ? 2 : dt == DType::Q8_0 ? 3
         : (dt == DType::Q4_0 && q4_0_tma_enabled()) ? 4 : -1;
}

int g_num_sms = 0;
int num_sms() {
    if (!g_num_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return g_num_sms;
}

constexpr size_t SMEM_CTA = 227 * 1024, SMEM_HALF = 113 * 1024;      // the most a CTA may have; the most of which two fit an SM

bool quarter_enabled() {          // NT_B200_GEMV_QB=1: opt-in A/B aid (measured slower)
    static const bool on = [] { const char* e = getenv("NT_B200_GEMV_QB"); return e && *e && !(e[0] == '0' && e[1] == 0); }();
    return on;
}

bool quarter_split_enabled() {    // NT_B200_GEMV_QB_SPLIT=0: launches that mix Q6_K with Q4_K/Q5_K stay one launch of the default kernel
    static const bool on = [] { const char* e = getenv("NT_B200_GEMV_QB_SPLIT"); return !(e && e[0] == '0' && e[1] == 0); }();
    return on;
}

// How the 16 warps of an SM are dealt out: CTAs of `teams` teams of `kw` warps, a ring of `stages` stages to a team.  stages == 0: no form fits.
struct TeamPlan { int kw, teams, stages, slot, planes; };
int team_slot(int mask, int kw) {         // bytes of a stage
    int slot = 0;
    for (int f = 0; f < 5; f++) if ((mask >> f) & 1 && MROWS * stage_pitch(f, kw) > slot) slot = MROWS * stage_pitch(f, kw);
    return slot;
}
TeamPlan plan_teams(int mask, int K, int groups, bool four) {
    auto form = [&](int kw, int teams, size_t cap) {
        TeamPlan t{kw, teams, 0, team_slot(mask, kw), 3};
        for (int planes = four ? 4 : 3; planes >= 3 && t.stages < 1; planes--) {      // four digits where that leaves a stage
            const size_t fixed = SM_X + x_bytes(K, planes);
            if (cap > fixed) t.stages = (int)std::min<size_t>(MAX_STAGES, (cap - fixed) / ((size_t)t.slot * teams));
            t.planes = planes;
        }
        return t;
    };
    // Teams of 4 share one copy of the vector and pay the meeting at the end of 16 rows half as often, four of them hide one another's barriers: the rule for
    // every launch that gives each SM more than a group (Q4_K 57344 x 8192 in a graph of its own: 45.5 us, 58 in teams of 8, 53.4 with the dp4a kernel that this
    // one replaced; cold and alone 50.6).
    // Fewer groups than SMs: more warps finish a group sooner, 8 (Q8_0 1024 x 4096: 4.8 us, 6.2 in teams of 4; Q4_K 4096 x 4096, 256 groups: 5.1 and 4.9), for
    // long rows 16 (Q6_K 1024 x 14336: 9.9 us, 11.0 in a team of 8, 12.2 before; Q8_0 2048 x 28672: 23.2, 29.7, 24.5); in between two teams of 8 in a CTA, since
    // the vector does not fit twice (Q4_K 4096 x 14336: 11.4 us, 12.3 in teams of 4, 16.9 before).
    TeamPlan t = K > 8192 ? (groups > 256 ? form(4, 4, SMEM_CTA) : groups > 148 ? form(8, 2, SMEM_CTA) : form(16, 1, SMEM_CTA))
                          : (groups > 148 ? form(4, 4, SMEM_CTA) : form(8, 1, SMEM_HALF));
    // Rings of one stage in four teams: two teams of 8 have the same bytes under way in stages of twice the columns, and half as many barriers, where they have two stages
    // (Q4_K 8192 x 28672: 36.3 us, 39.2 in teams of 4; Q5_K 8192 x 22016 call after call 31.9, 39.4) or are one round (Q8_0 4113 x 27904 35.6, 51.3); with one stage and more
    // rounds they are the slower ones (Q8_0 14529 x 27904 112.9 us, 103.8; Q6_K 14529 x 48128 224.5, 207.6).  Two stages in teams of 4 are the better of the two
    // (Q6_K 8192 x 28672: 46.6 us, 49.4 in teams of 8).
    if (t.kw == 4 && t.stages < 2 && K > 8192) {
        const TeamPlan u = form(8, 2, SMEM_CTA);
        if (u.stages >= 2 || groups <= 2 * 148 || u.planes > t.planes) t = u;      // (four digits: Q4_0 8192 x 36096 72 us, 1217 where the generic form takes it)
    }
    // Very long rows (from 41984 on, by format): the vector leaves no room for a stage of every team.  One team of 8 always has one.
    static const int ord[3][2] = {{8, 2}, {16, 1}, {8, 1}};
    for (int i = 0; t.stages < 1 && i < 3; i++) t = form(ord[i][0], ord[i][1], SMEM_CTA);
    return t;
}

// Gate and up as 8 rows of each to a group instead of two groups, where their rows can lie side by side in a stage and the last round then leaves fewer teams idle:
// 70B, 1792 pairs of groups over 592 teams are 3.03 rounds and cost four, 3584 groups of half the work 6.05 and cost seven (48.8 -> 45.9 us).  Where the number of rounds
// stays (8B: two, or four halves) pairs are no slower: 14.5 us, 14.9 in halves.
bool halves_of(const GemvMat& a, const GemvMat& b, int K) {
    auto pitch = [&](const GemvMat& m) { return m.row_pitch ? m.row_pitch : dtype_row_size(m.dtype, K); };
    const int pairs = (a.out + MROWS - 1) / MROWS, teams = MAX_TEAMS * std::max(1, num_sms());
    auto rounds = [&](int n) { return (n + teams - 1) / teams; };
    return fmt_of(a.dtype) == fmt_of(b.dtype) && pitch(a) == pitch(b) && rounds((a.out + 7) / 8) < 2 * rounds(pairs);
}

// format mixes with a kernel of their own
bool one_launch(int mask) { return mask == 1 || mask == 2 || mask == 4 || mask == 8 || mask == 3 || mask == 5 || mask == 16; }

template <int MASK, int KW, int TEAMS>
void launch_teams(KqParams& p, cudaStream_t s) {
    constexpr int ctas = SM_WARPS / (TEAMS * KW);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(gemv_mma_kernel<MASK, KW, TEAMS>, (int)SMEM_CTA, configured);
    const size_t smem = SM_X + x_bytes(p.K, MASK & WHOLE ? 4 : 3) + (size_t)p.stages * p.slot * TEAMS;
    const int places = num_sms() * (smem > SMEM_HALF ? 1 : ctas);
    launch_k_pdl(true, gemv_mma_kernel<MASK, KW, TEAMS>, dim3(p.total_groups < places ? p.total_groups : places), dim3(TEAMS * (KW + 1) * 32), smem, s, p);
    count_launch();
}

template <int MASK>
void launch_fmt(KqParams& p, cudaStream_t s) {
    constexpr int formats = MASK & ~WHOLE;
    int total = 0;
    for (int i = 0; i < p.n_mat; i++) { p.mat[i].groups = (p.mat[i].out + MROWS - 1) / MROWS; total += p.mat[i].groups; }
    p.total_groups = p.halves ? (p.mat[0].out + 7) / 8 : p.n_seg == 2 ? p.mat[0].groups : total;
    const TeamPlan t = plan_teams(formats, p.K, p.total_groups, MASK != formats);
    NT_CHECK(t.stages >= 1, "gemv_kq: shared memory budget exceeded");
    p.stages = t.stages; p.slot = t.slot;
    if constexpr (MASK != formats) if (t.planes == 3) { launch_fmt<formats>(p, s); return; }
    if (t.kw == 4) launch_teams<MASK, 4, 4>(p, s);
    else if (t.kw == 16) launch_teams<MASK, 16, 1>(p, s);
    else if (t.teams == 2) launch_teams<MASK, 8, 2>(p, s);
    else launch_teams<MASK, 8, 1>(p, s);
}

}  // namespace

int gemv_kq_format(DType dt) { return fmt_of(dt); }

// Rows of whole super-blocks that start on 16-byte boundaries: what the entries that answer with a code (nt_b200_gemv_fused*) accept.
bool gemv_kq_supported(const GemvMat* mats, int n_mat, int K) {
    if (!gemv_kq_any_pitch(mats, n_mat, K)) return false;
    for (int i = 0; i < n_mat; i++) {
        const size_t pitch = mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K);
        if (pitch & 15) return false;
    }
    return true;
}
// The kernel itself also takes rows at any even pitch (Q6_K rows of an odd number of super-blocks): it copies whole 16-byte units around a row.
bool gemv_kq_any_pitch(const GemvMat* mats, int n_mat, int K) {
    if (n_mat < 1 || n_mat > MAX_MATS || K % 256 != 0 || K <= 0 || K > MAX_K) return false;
    for (int i = 0; i < n_mat; i++) {
        const int f = fmt_of(mats[i].dtype);
        if (f < 0 || mats[i].out <= 0) return false;
        const size_t row = dtype_row_size(mats[i].dtype, K), pitch = mats[i].row_pitch ? mats[i].row_pitch : row;
        if ((reinterpret_cast<uintptr_t>(mats[i].W) & 15) || pitch < row || (pitch & (f == 2 ? 1 : 15))) return false;
    }
    int plan[4];
    return K <= 32768 || gemv_kq_plan(mats, n_mat, K, false, false, plan);      // up to there every form fits
}

// plan: warps of a team, teams of a CTA, stages of a team's ring, digits of an activation (the first matrix's where every matrix has a launch of its own)
bool gemv_kq_plan(const GemvMat* mats, int n_mat, int K, bool swiglu, bool whole, int* plan) {
    int mask = 0, groups = 0;
    for (int i = 0; i < n_mat; i++) { mask |= 1 << fmt_of(mats[i].dtype); groups += (mats[i].out + MROWS - 1) / MROWS; }
    if (!one_launch(mask)) {
        for (int i = n_mat - 1; i >= 0; i--) if (!gemv_kq_plan(&mats[i], 1, K, false, whole, plan)) return false;
        return true;
    }
    if (swiglu) groups = halves_of(mats[0], mats[1], K) ? (mats[0].out + 7) / 8 : (mats[0].out + MROWS - 1) / MROWS;
    const TeamPlan t = plan_teams(mask, K, groups, whole && mask == 16);
    plan[0] = t.kw; plan[1] = t.teams; plan[2] = t.stages; plan[3] = t.planes;
    return t.stages >= 1;
}

void gemv_kq(const GemvMat* mats, int n_mat, int K, const GemvInput& in, GemvEpilogue ep, cudaStream_t s) {
    NT_CHECK(gemv_kq_any_pitch(mats, n_mat, K), "gemv_kq: unsupported shape/dtype/alignment");
    NT_CHECK(ep != GEMV_PEER || (in.peer && n_mat == 1), "gemv_kq: GEMV_PEER needs GemvInput::peer and a single matrix");
    // Opt-in A/B (NT_B200_GEMV_QB=1): the quarter-block dp4a kernel (gemv_kquant_q.cu); launches that mix Q6_K with another format are split per
    // matrix for it.
    if (quarter_enabled() && gemv_kq_supported(mats, n_mat, K)) {
        int mask = 0;
        for (int i = 0; i < n_mat; i++) mask |= 1 << fmt_of(mats[i].dtype);
        const bool one_family = mask == 1 || mask == 2 || mask == 3 || mask == 4 || mask == 8 || mask == 16;
        if (one_family) {
            if (gemv_kq_quarter(mats, n_mat, K, in, ep, in.peer, s)) return;
        } else if (ep != GEMV_SWIGLU && ep != GEMV_PEER && quarter_split_enabled()) {
            // q/k (Q4_K) + v (Q6_K) of a Q4_K_M file: the Q4_K/Q5_K matrices in one launch, each Q6_K matrix in its own
            GemvMat fam[MAX_MATS];
            int nf = 0;
            for (int i = 0; i < n_mat; i++) if (mats[i].dtype != DType::Q6_K) fam[nf++] = mats[i];
            int fmask = 0;
            for (int i = 0; i < nf; i++) fmask |= 1 << fmt_of(fam[i].dtype);
            if (nf > 0 && (fmask == 1 || fmask == 2 || fmask == 3)) {
                bool ok = gemv_kq_quarter(fam, nf, K, in, ep, nullptr, s);
                for (int i = 0; i < n_mat && ok; i++)
                    if (mats[i].dtype == DType::Q6_K) ok = gemv_kq_quarter(&mats[i], 1, K, in, ep, nullptr, s);
                NT_CHECK(ok, "gemv_kq: the quarter-block kernel took part of a split launch only");
                return;
            }
        }
    }
    NT_CHECK((in.xq != nullptr) != (in.x != nullptr), "gemv_kq: exactly one of xq / x must be given");
    if (ep == GEMV_SWIGLU)
        NT_CHECK(n_mat == 2 && mats[0].out == mats[1].out, "gemv_kq: SWIGLU needs gate and up of equal rows");
    int mask = 0;
    for (int i = 0; i < n_mat; i++) mask |= 1 << fmt_of(mats[i].dtype);
    const bool plain = one_launch(mask);
    if (!plain && ep != GEMV_SWIGLU) {                         // rare mixes: one launch per matrix
        for (int i = 0; i < n_mat; i++) gemv_kq(&mats[i], 1, K, in, ep, s);
        return;
    }
    NT_CHECK(plain, "gemv_kq: SWIGLU over this format mix is not instantiated");
    KqParams p{};
    p.K = K; p.NB = K / 256;
    p.xq = static_cast<const int8_t*>(in.xq);
    p.x_f32 = in.x; p.norm_w = in.norm_w; p.eps = in.eps;
    if (ep == GEMV_PEER) p.peer = *in.peer;
    p.epilogue = (int)ep;
    p.n_mat = n_mat;
    for (int i = 0; i < n_mat; i++) {
        KqMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W);
        m.y = mats[i].y;
        m.out = mats[i].out;
        m.fmt = fmt_of(mats[i].dtype);
        m.row_pitch = (long long)(mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K));
    }
    p.halves = ep == GEMV_SWIGLU && halves_of(mats[0], mats[1], K);
    p.n_seg = ep == GEMV_SWIGLU && !p.halves ? 2 : 1;
    p.weights_settled = pdl_enabled();                         // a step of the engine; behind the launcher boundary the launch before may have written them
    p.status = wait_status();
    switch (mask) {
        case 1: launch_fmt<1>(p, s); break;
        case 2: launch_fmt<2>(p, s); break;
        case 4: launch_fmt<4>(p, s); break;
        case 3: launch_fmt<3>(p, s); break;
        case 8: launch_fmt<8>(p, s); break;
        case 16: if (in.whole) launch_fmt<16 | WHOLE>(p, s); else launch_fmt<16>(p, s); break;
        default: launch_fmt<5>(p, s); break;
    }
}

void gemv_kq_peer(const GemvMat& mat, int K, const GemvInput& in, const PeerOut& peer, cudaStream_t s) {
    NT_CHECK(mat.out == peer.hidden && peer.size >= 2 && peer.size <= PeerOut::kMaxTP, "gemv_kq_peer: rows must equal the exchanged vector length");
    GemvInput ip = in;
    ip.peer = &peer;
    gemv_kq(&mat, 1, K, ip, GEMV_PEER, s);
}

void gemv_kq(const GemvMat* mats, int n_mat, int K, const void* xq, GemvEpilogue ep, cudaStream_t s) {
    bool longer = ep != GEMV_PEER;
    for (int i = 0; i < n_mat; i++) longer = longer && gemv_xq_faster(mats[i], K);
    if (longer) { gemv_xq(mats, n_mat, K, xq, ep, s); return; }
    GemvInput in;
    in.xq = xq;
    gemv_kq(mats, n_mat, K, in, ep, s);
}

}}  // namespace nt::b200
