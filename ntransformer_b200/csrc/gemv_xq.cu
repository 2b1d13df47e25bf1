// gemv_xq.cu — GEMV over GGUF Q4_K / Q5_K / Q6_K / Q8_0 / Q4_0 blocks times an activation vector in pre-quantised form (kernels_internal.h "xq").
//
// Replaces reference kernels K2-K5 (src/cuda/gemm.cu:96-470) where the vector is quantised by a launch of its own: the decode step's unfused form, and long rows.  Its
// arithmetic, lane by lane and sum by sum, is the persistent decode-step kernel's GEMV phase (gemv_kq_device.cuh, engine/decode_megakernel.cu), so that
// the two forms of a decoded token can be compared: 22-bit activations, IDP.4A products, one F32 scale for 16 or 32 weights, chunks added in order.
//   * chunk-stationary warps: a row is cut into chunks of 16 super-blocks (4096 weights); warp w of a CTA owns chunk (w % NC) for the whole kernel, lane <->
//     one 128-weight half super-block, whose slice of the vector sits in registers;
//   * each warp streams its rows through a private ring of bulk copies: one stage = 4 rows x 16 super-blocks;
//   * the NC warps that hold the chunks of a row-group meet once per row-group and one of them adds the partial sums in a fixed order.
// Bound by instruction issue (2.0 instructions a weight; 57344 x 8192 in Q4_K 53 us): gemv_kquant.cu is faster but for long rows (gemv_xq_faster).
#include "kernels_internal.h"
#include "ring.cuh"
#include "wait_status.cuh"
#include "xquant.cuh"
#include "gemv_kq_device.cuh"
#include <cuda_fp16.h>

namespace nt { namespace b200 {

namespace {

constexpr int MAX_MATS = 3;
constexpr int MIN_WARPS = 4, MAX_WARPS = 12;

struct XqMat {
    const uint8_t* W;
    float* y;
    int out;
    int groups;        // ceil(out / RG)
    int fmt;           // 0 Q4_K, 1 Q5_K, 2 Q6_K, 3 Q8_0 (as groups of 8 blocks), 4 Q4_0 (likewise)
    long long row_pitch;
};
struct XqParams {
    XqMat mat[MAX_MATS];
    int n_mat;
    int K, NB, NC;             // elements, super-blocks per row, chunks per row (NC <= warps)
    const int8_t* xq;
    int total_groups;          // SWIGLU: groups of mat[0]
    int n_seg;                 // segments (matrices) per row-group: 2 for SWIGLU else 1
    int epilogue;
    int stages;                // ring depth per warp
    int gpc;                   // row-groups a CTA processes per round = warps / NC
    // Rounds over grid * gpc warp slots.  A last round that fills at most half (a quarter) of them deals its tail_groups row-groups out 2 (1) rows at a
    // time over all slots, so that it costs tail_nr / 4 of a round.  tail_nr == 4: no split.
    int full_rounds, tail_groups, tail_nr;
    unsigned* status;          // wait_status.cuh
};

// MASK: bit f set <=> matrices of format f may appear in this launch (mixed Q4_K_M projections share one launch).
template <int MASK, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS <= 6 ? 2 : 1) gemv_xq_kernel(const __grid_constant__ XqParams p) {
    constexpr int SLOT = RG * BS * max_blk(MASK);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float partial[2][MAX_WARPS][2][RG];      // [buffer][warp][segment][row]
    const int K = p.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stages = p.stages, NC = p.NC, NB = p.NB, n_seg = p.n_seg, gpc = p.gpc;
    // smem carve-up: [ring stage 0: WARPS slots][stage 1: WARPS slots]...[mbarriers]
    uint8_t* ring = smem + (size_t)warp * SLOT;                             // this warp's slot of stage s: ring + s * WARPS * SLOT
    constexpr size_t STAGE_STRIDE = (size_t)WARPS * SLOT;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)stages * STAGE_STRIDE) + warp * stages;

    const int chunk = warp % NC, gsub = warp / NC;        // this warp's chunk of every row, and its row-group slot
    const int n_rounds = p.full_rounds + (p.tail_groups > 0 ? 1 : 0);
    const int nbc = min(BS, NB - chunk * BS);              // super-blocks in this warp's chunk
    // what this warp slot holds in `round`: row-group g (global), the first row's offset inside it and the number of rows
    auto slot_of = [&](int round, int& g, int& row_sub, int& nr) -> bool {
        if (round < p.full_rounds || p.tail_nr >= RG) {
            g = (round * (int)gridDim.x + (int)blockIdx.x) * gpc + gsub; row_sub = 0; nr = RG;
            return g < p.total_groups;
        }
        nr = p.tail_nr;
        const int per = RG / nr, u = (int)blockIdx.x * gpc + gsub;
        g = p.full_rounds * (int)gridDim.x * gpc + u / per;
        row_sub = (u % per) * nr;
        return u < p.tail_groups * per;
    };
    auto locate = [&](int g, int seg, int& mi, int& gl) {  // matrix and local row-group of global group g
        if (n_seg == 2) { mi = seg; gl = g; return; }
        mi = 0;
        while (mi + 1 < p.n_mat && g >= p.mat[mi].groups) { g -= p.mat[mi].groups; mi++; }
        gl = g;
    };
    const int n_stages_total = n_rounds * n_seg;           // flattened stage index s = round * n_seg + seg
    int p_round = 0, p_seg = 0;                            // producer cursor (lane 0): the next stage to fetch
    auto issue_next = [&](int slot) {                      // lane 0: bulk copies of the next stage into ring slot
        uint64_t* bar = bars + slot;
        int g, row_sub, nr, mi = 0, gl = 0;
        bool have = slot_of(p_round, g, row_sub, nr);
        if (have) {
            locate(g, p_seg, mi, gl);
            have = gl * RG + row_sub < p.mat[mi].out;        // a slice of a ragged last group may hold no row
        }
        if (!have) {
            mbar_expect_tx(bar, 0);                          // nothing to fetch: just complete the phase
        } else {
            const XqMat& m = p.mat[mi];
            const int blkb = (MASK == 1) ? 144 : (MASK == 2) ? 176 : (MASK == 4) ? 210 : (MASK == 8) ? 272 : (MASK == 16) ? 144 : (m.fmt == 0 ? 144 : m.fmt == 1 ? 176 : 210);
            // copy size rounded up to 16 B (a 210-byte Q6_K tail may spill into row padding; checked on the host)
            const uint32_t bytes = ((uint32_t)(nbc * blkb) + 15u) & ~15u;
            mbar_expect_tx(bar, bytes * nr);
            uint8_t* dst = ring + (size_t)slot * STAGE_STRIDE;
            const int row0 = gl * RG + row_sub;
            const uint8_t* src = m.W + (long long)chunk * (BS * blkb) + (long long)row0 * m.row_pitch;
            for (int r = 0; r < nr; r++)                     // behind a ragged last group: its last row once more
                bulk_g2s(dst + r * (BS * blkb), src + (long long)min(r, m.out - 1 - row0) * m.row_pitch, bytes, bar);
        }
        if (++p_seg == n_seg) { p_seg = 0; p_round++; }
    };

    if (lane == 0) {
        for (int s = 0; s < stages; s++) mbar_init(bars + s, 1);
        mbar_fence_init();
    }
    __syncwarp();
    int issued = 0;
    if (lane == 0)                                           // weights do not depend on the previous kernel
        for (; issued < stages && issued < n_stages_total; issued++) issue_next(issued);
    pdl_wait();

    // ---- this lane's activation slice -> registers (once; planes stored with the 16-byte-column swizzle of xquant.cuh) ----
    const int blk = lane >> 1, h = lane & 1;
    const uint32_t hb = (uint32_t)((chunk * BS + min(blk, nbc - 1)) * 2 + h);   // global half-block index (clamped for idle lanes)
    XRegs X;
    {
        const int8_t* xq = p.xq;
        const uint32_t sw = (hb & 7u) << 4;
#pragma unroll
        for (int pl = 0; pl < 3; pl++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int4 v = __ldg(reinterpret_cast<const int4*>(xq + (size_t)pl * K + ((hb * 128u + 16u * i) ^ sw)));
                X.x[pl][4 * i] = v.x; X.x[pl][4 * i + 1] = v.y; X.x[pl][4 * i + 2] = v.z; X.x[pl][4 * i + 3] = v.w;
            }
        const float* fs = reinterpret_cast<const float*>(xq + 3 * (size_t)K);
        const float4 sv = __ldg(reinterpret_cast<const float4*>(fs + hb * 4));
        X.sx[0] = sv.x; X.sx[1] = sv.y; X.sx[2] = sv.z; X.sx[3] = sv.w;
        const float4 u0 = __ldg(reinterpret_cast<const float4*>(fs + K / 32 + hb * 8));
        const float4 u1 = __ldg(reinterpret_cast<const float4*>(fs + K / 32 + hb * 8 + 4));
        X.s16[0] = u0.x; X.s16[1] = u0.y; X.s16[2] = u0.z; X.s16[3] = u0.w;
        X.s16[4] = u1.x; X.s16[5] = u1.y; X.s16[6] = u1.z; X.s16[7] = u1.w;
    }
    pdl_launch_dependents();

    int slot = 0;
    uint32_t parity = 0;
    uint32_t tries = WAIT_TRIES;                                       // 0: a wait of this lane has run out
    for (int round = 0; round < n_rounds; round++) {
        int g, row_sub, nr;
        const bool live = slot_of(round, g, row_sub, nr);
        float res[2] = {0.f, 0.f};
        for (int seg = 0; seg < n_seg; seg++) {
            float acc[RG] = {0.f, 0.f, 0.f, 0.f};
            wait_phase(bars + slot, parity, p.status, tries);
            if (live && blk < nbc) {
                int mi, gl;
                locate(g, seg, mi, gl);
                const uint8_t* slot_base = ring + (size_t)slot * STAGE_STRIDE;
                const int fmt = (MASK == 1) ? 0 : (MASK == 2) ? 1 : (MASK == 4) ? 2 : (MASK == 8) ? 3 : (MASK == 16) ? 4 : p.mat[mi].fmt;
                if (nr == RG) {
                    if ((MASK & 1) && fmt == 0) process_stage<0>(slot_base, blk, h, X, acc);
                    if ((MASK & 2) && fmt == 1) process_stage<1>(slot_base, blk, h, X, acc);
                    if ((MASK & 4) && fmt == 2) process_stage<2>(slot_base, blk, h, X, acc);
                    if ((MASK & 8) && fmt == 3) process_stage<3>(slot_base, blk, h, X, acc);
                    if ((MASK & 16) && fmt == 4) process_stage<4>(slot_base, blk, h, X, acc);
                } else {                                     // tail stage of 1 or 2 rows: one row at a time
                    const int rowp = BS * ((fmt == 0 || fmt == 4) ? 144 : fmt == 1 ? 176 : fmt == 2 ? 210 : 272);
#pragma unroll 1
                    for (int r = 0; r < nr; r++) {
                        float a1[RG] = {0.f, 0.f, 0.f, 0.f};
                        const uint8_t* rb = slot_base + r * rowp;
                        if ((MASK & 1) && fmt == 0) process_stage<0, 1>(rb, blk, h, X, a1);
                        if ((MASK & 2) && fmt == 1) process_stage<1, 1>(rb, blk, h, X, a1);
                        if ((MASK & 4) && fmt == 2) process_stage<2, 1>(rb, blk, h, X, a1);
                        if ((MASK & 8) && fmt == 3) process_stage<3, 1>(rb, blk, h, X, a1);
                        if ((MASK & 16) && fmt == 4) process_stage<4, 1>(rb, blk, h, X, a1);
                        acc[0] = (r == 0) ? a1[0] : acc[0];       // no dynamic indexing: acc stays in registers
                        acc[1] = (r == 1) ? a1[0] : acc[1];
                    }
                }
            }
            __syncwarp();
            if (lane == 0 && issued < n_stages_total && tries) issue_next(slot);
            issued++;
            if (++slot == stages) { slot = 0; parity ^= 1u; }
            res[seg] = reduce4(acc, lane);
        }
        // ---- combine the NC chunk partials of each row-group (fixed order => deterministic) ----
        const int buf = round & 1;
        if (live && (lane & 7) == 0) {
            const int r = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
            partial[buf][warp][0][r] = tries ? res[0] : __uint_as_float(0x7FFFFFFFu);      // NaN
            partial[buf][warp][1][r] = res[1];
        }
        __syncthreads();
        if (live && chunk == 0 && lane < nr) {
            float v0 = 0.f, v1 = 0.f;
            for (int c = 0; c < NC; c++) {
                v0 += partial[buf][gsub * NC + c][0][lane];
                if (n_seg == 2) v1 += partial[buf][gsub * NC + c][1][lane];
            }
            int mi, gl;
            locate(g, 0, mi, gl);
            const XqMat& m = p.mat[mi];
            const int row = gl * RG + row_sub + lane;
            if (row < m.out) {
                if (p.epilogue == GEMV_SWIGLU) m.y[row] = __fdividef(v0, 1.0f + __expf(-v0)) * v1;      // gemm.cu:713-725's fast-math expression
                else if (p.epilogue == GEMV_ADD) m.y[row] += v0;
                else m.y[row] = v0;
            }
        }
    }
}

constexpr size_t SMEM_CAP = 227 * 1024 - 1024;    // static __shared__ counts against the cap

template <int MASK, int WARPS>
void launch_warps(XqParams& p, int sms, cudaStream_t s) {
    constexpr size_t SLOT = RG * BS * max_blk(MASK);
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(gemv_xq_kernel<MASK, WARPS>, (int)SMEM_CAP, configured);
    int grid = sms;
    const int slots = grid * p.gpc;
    p.full_rounds = p.total_groups / slots;
    p.tail_groups = p.total_groups % slots;
    p.tail_nr = p.tail_groups == 0 ? RG : 4 * p.tail_groups <= slots ? 1 : 2 * p.tail_groups <= slots ? 2 : RG;
    if (p.full_rounds == 0) {                                  // fewer units than warp slots: no more CTAs than there is work
        const int need = (p.tail_groups * (RG / p.tail_nr) + p.gpc - 1) / p.gpc;
        if (need < grid) grid = need;
    }
    launch_k(gemv_xq_kernel<MASK, WARPS>, dim3(grid), dim3(WARPS * 32), (size_t)WARPS * p.stages * (SLOT + 8) + 128, s, p);
    count_launch();
}

// Warps of a CTA: the largest multiple of NC (chunks per row) in [MIN_WARPS, MAX_WARPS] with two stages each, or with one.
template <int MASK>
void launch_fmt(XqParams& p, int sms, cudaStream_t s) {
    constexpr size_t SLOT = RG * BS * max_blk(MASK), budget = SMEM_CAP - 256;
    int w = 0;
    for (int least = 2; least >= 1 && !w; least--)
        for (int n = p.NC; n <= MAX_WARPS; n += p.NC)
            if (n >= MIN_WARPS && (size_t)n * least * (SLOT + 8) <= budget) w = n;
    NT_CHECK(w != 0, "gemv_xq: shared memory budget exceeded");
    p.gpc = w / p.NC;
    p.stages = (int)(budget / ((size_t)w * (SLOT + 8)));
    if (p.stages > 4) p.stages = 4;
    switch (w) {
        case 12: launch_warps<MASK, 12>(p, sms, s); break;
        case 11: launch_warps<MASK, 11>(p, sms, s); break;
        case 10: launch_warps<MASK, 10>(p, sms, s); break;
        case 9: launch_warps<MASK, 9>(p, sms, s); break;
        case 8: launch_warps<MASK, 8>(p, sms, s); break;
        case 7: launch_warps<MASK, 7>(p, sms, s); break;
        case 6: launch_warps<MASK, 6>(p, sms, s); break;
        case 5: launch_warps<MASK, 5>(p, sms, s); break;
        default: launch_warps<MASK, 4>(p, sms, s); break;
    }
}

}  // namespace

bool gemv_xq_supported(const GemvMat* mats, int n_mat, int K) {
    if (n_mat < 1 || n_mat > MAX_MATS || K % 256 != 0 || K <= 0) return false;
    const int NB = K / 256, NC = (NB + BS - 1) / BS;
    if (NC > MAX_WARPS) return false;              // one warp per chunk of a row (K <= 49152)
    for (int i = 0; i < n_mat; i++) {
        if (gemv_kq_format(mats[i].dtype) < 0 || mats[i].out <= 0) return false;
        const size_t pitch = mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K);
        if ((reinterpret_cast<uintptr_t>(mats[i].W) & 15) || (pitch & 15)) return false;
        // the last chunk of a row is copied in 16-byte units and must stay inside the row pitch
        const size_t blk = dtype_row_size(mats[i].dtype, 256);     // bytes per 256 weights
        const int last = NB - (NC - 1) * BS;
        if ((size_t)(NC - 1) * BS * blk + ((last * blk + 15) & ~(size_t)15) > pitch) return false;
    }
    return true;
}

// Long rows: beside the vector (3.25 bytes an element) gemv_kquant.cu has one or two ring stages to a team, this kernel all of shared memory.  The line lies where
// that kernel is down to one stage of one super-block to a warp (Q8_0 from 26624 columns, Q6_K from 35328), and at 32768 for the formats whose stage holds two.
// Decode steps of three layers, the down projection here against there (its quantise launch included): Q8_0 20480 wide 457 us against 460, 24576 550 / 545, 28672
// 760 / 807; Q6_K 24576 557 / 547, 28672 757 / 755, 32768 781 / 788, 36864 835 / 896; Q4_K 18944 (four layers) 326 / 320, 24576 496 / 506, 28672 554 / 557, 32768
// 564 / 573, 36864 829 / 877, 40960 608 / 635, 49152 666 / 802; Q5_K 24576 469 / 462, 28672 611 / 616, 40960 701 / 718.  70B in Q4_K_M (28672) 94.8 tok/s against 95.4.
bool gemv_xq_faster(const GemvMat& m, int K) {
    if (K < 20480 || !gemv_xq_supported(&m, 1, K)) return false;
    int plan[4];
    const bool single = m.dtype == DType::Q6_K || m.dtype == DType::Q8_0;
    return K >= 32768 || !gemv_kq_any_pitch(&m, 1, K) || (single && gemv_kq_plan(&m, 1, K, false, false, plan) && plan[2] == 1);
}

void gemv_xq(const GemvMat* mats, int n_mat, int K, const void* xq, GemvEpilogue ep, cudaStream_t s) {
    NT_CHECK(gemv_xq_supported(mats, n_mat, K) && ep != GEMV_PEER, "gemv_xq: unsupported shape/dtype/alignment");
    NT_CHECK(ep != GEMV_SWIGLU || (n_mat == 2 && mats[0].out == mats[1].out), "gemv_xq: SWIGLU needs gate and up of equal rows");
    int mask = 0;
    for (int i = 0; i < n_mat; i++) mask |= 1 << gemv_kq_format(mats[i].dtype);
    const bool plain = (mask & (mask - 1)) == 0 || mask == 3 || mask == 5;
    if (!plain && ep != GEMV_SWIGLU) {                         // rare mixes: one launch per matrix
        for (int i = 0; i < n_mat; i++) gemv_xq(&mats[i], 1, K, xq, ep, s);
        return;
    }
    NT_CHECK(plain, "gemv_xq: SWIGLU over this format mix is not instantiated");
    XqParams p{};
    p.K = K; p.NB = K / 256; p.NC = (p.NB + BS - 1) / BS;
    p.xq = static_cast<const int8_t*>(xq);
    p.epilogue = (int)ep;
    p.n_mat = n_mat;
    int total = 0;
    for (int i = 0; i < n_mat; i++) {
        XqMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W);
        m.y = mats[i].y;
        m.out = mats[i].out;
        m.groups = (mats[i].out + RG - 1) / RG;
        m.fmt = gemv_kq_format(mats[i].dtype);
        m.row_pitch = (long long)(mats[i].row_pitch ? mats[i].row_pitch : dtype_row_size(mats[i].dtype, K));
        total += m.groups;
    }
    p.n_seg = ep == GEMV_SWIGLU ? 2 : 1;
    p.total_groups = p.n_seg == 2 ? p.mat[0].groups : total;
    p.status = wait_status();
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    switch (mask) {
        case 1: launch_fmt<1>(p, sms, s); break;
        case 2: launch_fmt<2>(p, sms, s); break;
        case 4: launch_fmt<4>(p, sms, s); break;
        case 3: launch_fmt<3>(p, sms, s); break;
        case 8: launch_fmt<8>(p, sms, s); break;
        case 16: launch_fmt<16>(p, sms, s); break;
        default: launch_fmt<5>(p, sms, s); break;
    }
}

}}  // namespace nt::b200
