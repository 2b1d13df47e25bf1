// attention_prefill_tc.cu — causal GQA attention of a run of prompt tokens over the F16 cache on the 5th-generation tensor cores (tcgen05), sm_100a.
//
// Same contract as the reference's attention_prefill_kernel (src/cuda/attention.cu:216-311): F32 queries [seq][n_heads][hd], F16 cache [max_seq][n_kv][hd], query i
// attends keys 0..start_pos + i.  The form on mma.sync (attention_prefill_mma.cu), which windows and BF16 caches still take, is bound by that instruction: two halves
// of each query and of each weight make four products where two are counted.  Here:
//   * a CTA owns two tiles of 128 queries that share their keys (two heads of a key head; two runs of queries where it has an odd number): while the tensor cores
//     multiply for one, eight warps form the weights of the other (half of a row's keys each);
//   * scores S = (q_hi + q_lo) . K^T: queries split in shared memory, each row under a power of two that keeps its low halves' bits, keys by TMA, 128 at a time, two
//     buffers; 128 x 128 scores in tensor memory, three buffers that the tiles use in turn, so that a tile's next scores are there when its weights are handed over;
//   * weights exp2(f S - m) as F16 hi + lo take the scores' place in tensor memory, which is the A operand of (p_hi + p_lo) . V;
//   * that product of 128 keys starts at zero in the fourth quarter of tensor memory and is taken from there at once; the rows' sums are kept in F32 registers,
//     rescaled there where the maximum moves.
// 1000 tokens behind 1023, 32 heads of 128 over 8: 174 us on mma.sync, 62.2 here with eight warps for the weights, 56.9 with sixteen; 50 GFLOP issued in it, 0.9 PFLOP/s.
// Bound by the forming of the weights, behind which the tensor cores wait.
#include "kernels_internal.h"
#include "ring.cuh"
#include "tc_device.cuh"
#include "attention_row.cuh"
#include "wait_status.cuh"
#include <cuda.h>
#include <cuda_fp16.h>

namespace nt { namespace b200 {

namespace {

constexpr int TQ = 128, TK = 128;                        // queries of a tile, keys of a step
constexpr int TC_THREADS = 20 * 32;                      // warps 0-7 and 8-15: softmax of the two tiles, 16: TMA, 17: MMA; registers 4 x 104 + 64 = 5 x 96 at launch
template <int HD> struct TcSmem {
    static constexpr int Q = TQ * HD * 2, KV = TK * HD * 2;              // bytes of a tile's half of the queries; of a step's keys or values
    static constexpr int K0 = 4 * Q, V0 = K0 + 2 * KV, ALL = V0 + KV;
};

// Values as the B operand: N (channels) contiguous, SWIZZLE_128B: 64 channels x 8 keys to an atom of 1024 bytes, the next 8 keys 1024 bytes on (stride offset), the
// next 64 channels a whole box on (leading offset)
__device__ __forceinline__ uint64_t make_desc_mn(const void* smem_ptr, uint32_t box_bytes) {
    const uint64_t addr = (uint64_t)(smem_u32(smem_ptr) & 0x3FFFFu) >> 4;
    return addr | ((uint64_t)(box_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

struct TcAttn {
    float* out;
    const float* Q;
    const __half *kc, *vc;
    int seq_len, start_pos, n_heads, n_kv, pairs_of_queries;      // pairs_of_queries: a key head has an odd number of heads
    float scale;
    unsigned* status;
};

template <int HD>
__global__ void __launch_bounds__(TC_THREADS, 1) prefill_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ TcAttn p) {
    using S = TcSmem<HD>;
    constexpr int BOXES = HD / 64, BOX = TK * 128;                // boxes of 64 channels
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;                                     // the declared alignment: there is no room to round up
    if (smem_u32(smem) & 1023u) { if (threadIdx.x == 0) report(p.status); return; }
    __shared__ uint64_t k_full[2], k_empty[2], v_full, v_empty, q_full, s_full[3], p_full[2], o_full[2], o_empty;
    __shared__ float row_word[2][2 * TQ];                         // [half of the keys][row]: factors first, then a step's maxima, at the end the sums
    __shared__ uint32_t tmem_base_smem, dead_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t dead = smem_u32(&dead_smem);
    // the longest runs of keys first
    const int qt = (int)gridDim.x - 1 - (int)blockIdx.x, h0 = p.pairs_of_queries ? (int)blockIdx.y : 2 * (int)blockIdx.y, kvh = h0 / (p.n_heads / p.n_kv);
    const int first_q = qt * (p.pairs_of_queries ? 2 * TQ : TQ), last_q = min(first_q + (p.pairs_of_queries ? 2 * TQ : TQ), p.seq_len) - 1;
    const int n = (p.start_pos + last_q) / TK + 1;               // steps
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) { mbar_init(k_full + i, 1); mbar_init(k_empty + i, 1); mbar_init(p_full + i, 8); mbar_init(o_full + i, 1); }
        for (int i = 0; i < 3; i++) mbar_init(s_full + i, 1);
        mbar_init(&v_full, 1); mbar_init(&v_empty, 1); mbar_init(&q_full, 16); mbar_init(&o_empty, 8);
        dead_smem = 0;
        mbar_fence_init();
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_launch_dependents();
    pdl_wait();
    // Step j of tile t is item 2 j + t.  Tensor memory is this CTA's whole: an item's scores, then weights, at column 128 (item mod 3), its product with V at 384.

    if (warp < 16) {
        // ---- softmax: a row to two lanes, each with half of a step's keys and half of the channels (four warps to a scheduler hide what one waits for) ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        constexpr int HK = TK / 2, HC = HD / 2;
        const int t = warp >> 3, quarter = warp & 3, half = (warp >> 2) & 1, r = quarter * 32 + lane, head = p.pairs_of_queries ? h0 : h0 + t;
        const int q0 = first_q + (p.pairs_of_queries ? t * TQ : 0), row = q0 + r;
        const float* queries = behind_wait(p.Q);
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16, to = lanes + 384 + half * HC;
        uint8_t* mine = smem + 2 * t * S::Q;                      // the tile's queries
        {
            // a row to LR lanes, so that loads are whole lines; 4 channels to a lane
            constexpr int LR = HD / 4, RI = 32 / LR;              // lanes of a row, rows of an instruction
            const int c = lane % LR;
#pragma unroll 8
            for (int i = 0; i < 16 / RI; i++) {
                const int rr = quarter * 32 + half * 16 + i * RI + lane / LR;
                const float4 x = __ldg(reinterpret_cast<const float4*>(queries + ((size_t)min(q0 + rr, p.seq_len - 1) * p.n_heads + head) * HD) + c);
                float amax = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w)));
#pragma unroll
                for (int s = LR / 2; s > 0; s >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, s));
                const uint32_t e = __float_as_uint(amax) >> 23 & 255u;       // not finite, or zero: as it is
                const uint32_t up = e == 255u || e == 0u ? 127u : min(227u, max(27u, 264u - e));       // to 2^10 .. 2^11
                const float g = copysignf(__uint_as_float(up << 23), p.scale);        // the scale's sign goes with the queries: the greatest score stays the greatest
                // never zero: masked scores are -inf times it, and others as small as that have equal weights
                const float fq = fabsf(p.scale) * 1.4426950408889634f * __uint_as_float((254u - up) << 23);
                if (c == 0) row_word[0][t * TQ + rr] = fq == 0.f ? 1.1754944e-38f : fq;
                uint2 h, l;
                split_pair(x.x * g, x.y * g, 0, h.x, l.x);
                split_pair(x.z * g, x.w * g, 0, h.y, l.y);
                // 64 channels to a 128-byte swizzle row
                uint8_t* d = mine + (c >> 4) * (TQ * 128) + rr * 128 + ((((c & 15) >> 1) ^ (rr & 7)) << 4) + (c & 1) * 8;
                *reinterpret_cast<uint2*>(d) = h;
                *reinterpret_cast<uint2*>(d + S::Q) = l;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_full);
        }
        auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quarter) : "memory"); };      // the two warps of a quarter's rows
        meet();
        const float f = row_word[0][t * TQ + r];                  // of the row's scores: log2 e * scale, and the power of two taken back
        meet();
        uint64_t o[HC / 2];                                       // pairs of channels
#pragma unroll
        for (int i = 0; i < HC / 2; i++) o[i] = 0;
        float m = -INFINITY, l = 0.f;
        uint32_t ts = lanes + t * 128;                            // of the step's scores
#pragma unroll 1
        for (int j = 0; j < n; j++) {
            const int seen = p.start_pos + row - j * TK - half * HK;     // of this lane's keys those up to here are seen
            const bool whole = j * TK + TK - 1 <= p.start_pos + q0;      // by every row of the tile
            wait_cta(s_full + ((2 * j + t) % 3), ((2 * j + t) / 3) & 1, dead);      // (of the buffer: a tile's next scores may come before these are looked at)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < HK / 16; c++) {
                uint32_t v[16];
                tmem_ld16(ts + half * HK + 16 * c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (whole) {
#pragma unroll
                    for (int i = 0; i < 16; i++) mx = fmaxf(mx, __uint_as_float(v[i]));
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) mx = fmaxf(mx, 16 * c + i <= seen ? __uint_as_float(v[i]) : -INFINITY);
                }
            }
            row_word[half][t * TQ + r] = mx;                      // (the other warp has read the step before: that step's product waited for its weights)
            meet();
            mx = fmaxf(mx, row_word[half ^ 1][t * TQ + r]);
            const float mn = fmaxf(m, mx * f), base = mn == -INFINITY ? 0.f : mn, alpha = exp2f(m - base);      // (a run of keys wholly unseen leaves the maximum; step 0 has key 0)
            m = mn;
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < HK / 16; c++) {                   // 16 keys: 8 columns hi, 8 lo, where their scores were
                uint32_t v[16], w[16];
                tmem_ld16(ts + half * HK + 16 * c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!whole)
#pragma unroll
                    for (int i = 0; i < 16; i++) v[i] = 16 * c + i <= seen ? v[i] : 0xFF800000u;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float a = exp2f(fmaf(__uint_as_float(v[2 * i]), f, -base)), b = exp2f(fmaf(__uint_as_float(v[2 * i + 1]), f, -base));
                    sum += a + b;
                    split_pair(a, b, 0, w[i], w[8 + i]);
                }
                tmem_st16(ts + half * HK + 16 * c, w);
            }
            l = fmaf(l, alpha, sum);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + t);
            // the step's product joins the sums
            wait_cta(o_full + t, j & 1, dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t aa = pack2(alpha, alpha);
#pragma unroll
            for (int c = 0; c < HC / 16; c++) {
                uint32_t v[16];
                tmem_ld16(to + 16 * c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 8; i++) o[8 * c + i] = fma2(o[8 * c + i], aa, pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_empty);
            ts = ts == lanes ? lanes + 256 : ts - 128;            // two items on
        }
        row_word[half][t * TQ + r] = l;
        meet();
        if (word_set(dead)) report(p.status);
        else {
            // 16 rows at a time over the tile's queries (no product reads them any more), then whole lines to memory
            l += row_word[half ^ 1][t * TQ + r];
            const float inv = 1.0f / l;
            uint64_t odd = 0;                                     // NaN where a sum is infinite or NaN
#pragma unroll
            for (int i = 0; i < HC / 2; i++) odd = fma2(o[i], 0, odd);
            float odd0, odd1;
            unpack2(odd, odd0, odd1);
            unsigned again = __ballot_sync(0xFFFFFFFFu, row < p.seq_len && !(odd0 + odd1 == 0.f) && l < INFINITY);      // (a row that sees a NaN or infinite score is NaN)
            constexpr int PITCH = HC + 4, LR = HC / 4, RI = 32 / LR;
            float* stage = reinterpret_cast<float*>(mine) + (warp & 7) * 16 * PITCH;
#pragma unroll
            for (int part = 0; part < 2; part++) {
                if ((lane >> 4) == part)
#pragma unroll
                    for (int i = 0; i < HC / 4; i++) {
                        float4 x;
                        unpack2(o[2 * i], x.x, x.y); unpack2(o[2 * i + 1], x.z, x.w);
                        *reinterpret_cast<float4*>(stage + (lane & 15) * PITCH + 4 * i) = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
                    }
                __syncwarp();
#pragma unroll 4
                for (int i = 0; i < 16 / RI; i++) {
                    const int rr = i * RI + lane / LR, at = q0 + quarter * 32 + part * 16 + rr;
                    if (at < p.seq_len)
                        *(reinterpret_cast<float4*>(p.out + ((size_t)at * p.n_heads + head) * HD + half * HC) + lane % LR) = *reinterpret_cast<const float4*>(stage + rr * PITCH + 4 * (lane % LR));
                }
                __syncwarp();
            }
            for (; again; again &= again - 1) row_alone<HD, HC>(p, q0 + quarter * 32 + __ffs(again) - 1, head, half * HC, lane);
        }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 16) {
        if (lane == 0) {                                          // ---- keys and values by TMA: keys a step ahead ----
            auto load = [&](uint8_t* d, const CUtensorMap* map, int j, uint64_t* full) {
                mbar_expect_tx(full, S::KV);
#pragma unroll
                for (int i = 0; i < BOXES; i++) tma_load_2d(d + i * BOX, map, kvh * HD + 64 * i, j * TK, full);
            };
            int keys = 1, values = 0;                             // steps whose keys, whose values are under way
            bool gone = false;
            load(smem + S::K0, &map_k, 0, k_full);
            for (int j = 0; j < n && !gone; j++) {
                if (j + 1 < n) {
                    wait_cta(k_empty + ((j + 1) & 1), (((j + 1) >> 1) & 1) ^ 1, dead);
                    if (!(gone = word_set(dead))) { load(smem + S::K0 + ((j + 1) & 1) * S::KV, &map_k, j + 1, k_full + ((j + 1) & 1)); keys = j + 2; }
                }
                wait_cta(&v_empty, (j & 1) ^ 1, dead);
                if (!(gone = gone || word_set(dead))) { load(smem + S::V0, &map_v, j, &v_full); values = j + 1; }
            }
            if (gone) {                                           // given up: the copies in flight
                for (int j = max(0, keys - 2); j < keys; j++) wait_flight(k_full + (j & 1), (j >> 1) & 1);
                if (values) wait_flight(&v_full, (values - 1) & 1);
            }
        }
    } else if (warp == 17) {
        // ---- MMA: the whole warp walks the loop and one lane issues by predicate, so that operands stay in uniform registers ----
        const uint32_t lead = elect_lane();
        constexpr uint32_t F32_M128 = (1u << 4) | (8u << 24);
        constexpr uint32_t IDESC_S = F32_M128 | ((uint32_t)(TK >> 3) << 17), IDESC_O = F32_M128 | ((uint32_t)(HD >> 3) << 17) | (1u << 16);      // V: N-major
        const uint64_t dq = make_desc(smem), dk = make_desc(smem + S::K0), dv = make_desc_mn(smem + S::V0, BOX);
        uint32_t sb = 0;                                          // columns of the next item's scores
        auto scores = [&](int item) {
            const int t = item & 1, j = item >> 1;
            if (t == 0) { wait_cta(k_full + (j & 1), (j >> 1) & 1, dead); asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
            const uint64_t a = dq + (uint64_t)(t * (2 * S::Q >> 4)), b = dk + (uint64_t)((j & 1) * (S::KV >> 4));
#pragma unroll
            for (int part = 1; part >= 0; part--)                 // the low halves first
#pragma unroll
                for (int s = 0; s < HD / 16; s++) {
                    const uint64_t at = (uint64_t)((s >> 2) * (TQ * 128 >> 4) + 2 * (s & 3));
                    umma_ss_by(lead, sb, a + (uint64_t)((part * S::Q) >> 4) + at, b + at, IDESC_S, part == 0 || s > 0);
                }
            umma_commit_by(lead, s_full + (sb >> 7));
            if (t == 1) umma_commit_by(lead, k_empty + (j & 1));
            sb = sb == 256 ? 0 : sb + 128;
        };
        wait_cta(&q_full, 0, dead);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        scores(0);
        scores(1);
        if (n > 1) scores(2);
#pragma unroll 1
        for (int item = 0; item < 2 * n; item++) {
            const int t = item & 1, j = item >> 1;
            const uint32_t pb = n > 1 ? sb : item * 128;          // the buffer used longest ago (three items are under way; with one step two)
            wait_cta(p_full + t, j & 1, dead);
            if (t == 0) wait_cta(&v_full, j & 1, dead);
            if (item > 0) wait_cta(&o_empty, (item - 1) & 1, dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int part = 1; part >= 0; part--)
#pragma unroll
                for (int s = 0; s < TK / 16; s++)
                    umma_ts_by(lead, 384, pb + 16 * s + 8 * part, dv + (uint64_t)(s * (2048 >> 4)), IDESC_O, part == 0 || s > 0);
            umma_commit_by(lead, o_full + t);
            if (t == 1) umma_commit_by(lead, &v_empty);
            if (item + 3 < 2 * n) scores(item + 3);               // (behind the product that read the buffer)
            else sb = sb == 256 ? 0 : sb + 128;
        }
        wait_flight(&v_empty, (n - 1) & 1);                       // the last commit: nothing of this CTA is in flight behind its end
    }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    if (warp == 17) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_smem), "n"(512));
}

template <int HD>
void launch_tc(const CUtensorMap& map_k, const CUtensorMap& map_v, const TcAttn& p, cudaStream_t s) {
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(prefill_tc_kernel<HD>, TcSmem<HD>::ALL, configured);
    const int rows = p.pairs_of_queries ? 2 * TQ : TQ;
    launch_k_pdl(true, prefill_tc_kernel<HD>, dim3((p.seq_len + rows - 1) / rows, p.pairs_of_queries ? p.n_heads : p.n_heads / 2), dim3(TC_THREADS), TcSmem<HD>::ALL, s, map_k, map_v, p);
    count_launch();
}

}  // namespace

// Whether this form takes a call: widths, pointers on 16 bytes, and positions inside the cache (its maps have a row for every key; the form on mma.sync stays inside
// a cache of max_seq rows whatever the positions)
bool attention_prefill_tc_takes(const float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads, int n_kv, int hd, int max_seq) {
    return seq_len >= 1 && (hd == 64 || hd == 128) && n_kv >= 1 && n_heads % n_kv == 0 && n_heads <= 65535 && start_pos >= 0 && (long long)start_pos + seq_len <= max_seq &&
           ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;
}

// A call that attention_prefill_tc_takes; false: nothing launched
bool attention_prefill_tc(float* out, const float* Q, const void* kc, const void* vc, int seq_len, int start_pos, int n_heads, int n_kv, int hd, float scale, cudaStream_t s) {
    // the maps end with the last key: rows of the cache behind it are zeros, whatever they hold
    CUtensorMap map_k, map_v;
    const uint64_t keys = (uint64_t)start_pos + seq_len, row = (uint64_t)n_kv * hd;
    if (!tc_map_f16(&map_k, kc, keys, row, TK) || !tc_map_f16(&map_v, vc, keys, row, TK)) return false;
    TcAttn p{out, Q, static_cast<const __half*>(kc), static_cast<const __half*>(vc), seq_len, start_pos, n_heads, n_kv, (n_heads / n_kv) % 2, scale, wait_status()};
    if (hd == 128) launch_tc<128>(map_k, map_v, p, s);
    else launch_tc<64>(map_k, map_v, p, s);
    return true;
}

}}  // namespace nt::b200
