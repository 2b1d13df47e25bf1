// prefill_dense.cu — tensor-core GEMM of some tokens over F16 or BF16 matrices: Y[T, N] (+)= X[T, K] . W[N, K]^T where tokens are few.
//
// The reference runs its GEMV once for each token (src/model/attention.cpp:144-162, ffn.cpp:96-133).  prefill_gemm.cu's tiles of 128 tokens x 256 rows leave most SMs idle there: the o
// projection of an 8B model over 100 tokens has 16 of them.  Here W is A (128 rows to a tile), tokens are B (NT, a multiple of 16 up to 128), and tiles times units of 256
// columns are dealt out evenly (tile_deal.cuh), so that every SM streams W.
//   * W and tokens by TMA into a ring of k-blocks of 64 columns, deep enough for HBM's latency (64 to 112 KB of W in flight to an SM);
//   * tokens as two halves (or two BF16), a unit of 256 columns to an accumulator, added up in F32 registers; or, in the fine form, as three (24 bits
//     and more, in small first parts: TokenParts) with 64 columns to an accumulator, as exact as F32 products one by one (the tensor cores cut off each addition, which leaves 1.86e-8 of a sum for each);
//   * the parts of a tile lie one behind the other in shared memory and are ONE operand of parts * NT rows: a product for 16 columns in place of two or three, and the epilogue adds
//     what the parts gave (21 tokens, 28672 x 4096, fine: 56.9 us with a product for each, 49.8 so).
// Bound by HBM where tokens are few (21 tokens, F16, with their split: gate and up of an 8B model 28672 x 4096 50 us, 4.7 TB/s; 4096 x 14336 40 us, of which 12 go to start, tail and
// shares), by L2 from 100 or so on (48 KB to a k-block for 512 cycles of products).  Before: 12 tokens of an F16 model (2 layers of 4096) one by one 3316 us, 379; tiles of 128 x 256
// over 100 tokens: 4096 x 4096 54 us, 29; 4096 x 14336 177, 50; over 300: 183, 91.  Error against 64 bits, 4096 columns: fine 1.0e-7 (one by one 1.6e-7), otherwise 3.5e-7 (9.7e-6
// with 4096 columns to an accumulator); BF16 1.0e-7 and 2.5e-6 (16 bits of an activation).
#include "kernels_internal.h"
#include "ring.cuh"
#include "tc_device.cuh"
#include "tile_deal.cuh"
#include "wait_status.cuh"
#include <cuda.h>
#include <algorithm>

namespace nt { namespace b200 {

namespace {

constexpr int KB = 64, W_TILE = 128 * KB * 2, STAGES_MAX = 8, BUFS_MAX = 8, THREADS = 12 * 32;      // warp 0 tokens, 1 MMA, 2 W, 4-11 epilogue
constexpr int NT_MAX = 128, NT_FINE = 80;                // tokens of a tile: parts * NT are an operand of 256 rows at most
constexpr size_t SMEM_CAP = 220 * 1024;

struct alignas(64) DenseMaps { CUtensorMap x, w[3]; };
struct DenseParams : Deal { int Mp, stages, stage, d_bufs, bf16; unsigned* status; };

template <int PARTS>
__global__ void __launch_bounds__(THREADS, 1) gemm_dense_tc_kernel(const __grid_constant__ DenseMaps maps, const __grid_constant__ DenseParams p) {
    constexpr int KC = PARTS == 3 ? 1 : 4;                         // k-blocks to an accumulator
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[STAGES_MAX], empty[STAGES_MAX], d_full[BUFS_MAX], d_empty[BUFS_MAX];
    __shared__ uint32_t tmem_base_smem, last_smem, dead_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NT = p.NT;
    const uint32_t b_tile = (uint32_t)NT * 128, stage = (uint32_t)p.stage, dead = smem_u32(&dead_smem);
    const int u0 = first_unit(p, blockIdx.x), u1 = first_unit(p, blockIdx.x + 1);
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.stages; i++) { mbar_init(full + i, 2); mbar_init(empty + i, 1); }      // tokens and W
        for (int i = 0; i < p.d_bufs; i++) { mbar_init(d_full + i, 1); mbar_init(d_empty + i, 8); }
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
    // W depends on no launch in flight: its copies start at once, tokens and everything written wait for the launch before
    pdl_launch_dependents();

    if (warp == 0 || warp == 2) {
        if (lane == 0) {                                           // ---- tokens, W by TMA ----
            uint32_t st = 0, par = 1, filled = 0;
            Place q = start(p, u0);
            if (warp == 0) pdl_wait();
            for (int u = u0; u < u1; u++, next(p, q)) {
                for (int kb = 0; kb < 4; kb++) {
                    wait_cta(empty + st, par, dead);
                    if (word_set(dead)) {
                        for (uint32_t s = 0; s < filled; s++) wait_flight(full + s, s < st ? par ^ 1u : par);      // the copies in flight
                        u = u1;
                        break;
                    }
                    filled = min(filled + 1, (uint32_t)p.stages);
                    uint8_t* d = smem + (size_t)st * stage;
                    const int k = q.b * 256 + kb * KB;
                    if (warp == 2) {
                        mbar_expect_tx(full + st, W_TILE);
                        tma_load_2d(d, &maps.w[q.mi], k, q.row0, full + st);
                    } else {
                        mbar_expect_tx(full + st, PARTS * b_tile);
#pragma unroll
                        for (int i = 0; i < PARTS; i++) tma_load_2d(d + W_TILE + i * b_tile, &maps.x, k, i * p.Mp + q.t0, full + st);      // a part lies Mp rows below the one before
                    }
                    if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA: the whole warp walks the loop, one lane issues ----
        const uint32_t lead = elect_lane();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(PARTS * NT >> 3) << 17) | (8u << 24) | (p.bf16 ? ((1u << 7) | (1u << 10)) : 0u);
        const uint64_t desc0 = make_desc(smem), stage_step = (uint64_t)(stage >> 4);
        uint32_t st = 0, par = 0, db = 0, dpar = 1;
        int last = -1;                                             // stage and parity of the last commit
        for (int u = u0; u < u1; u++) {
#pragma unroll 1
            for (int kb = 0; kb < 4; kb++) {
                const uint32_t d = db * PARTS * NT;
                if (kb % KC == 0) wait_cta(d_empty + db, dpar, dead);
                wait_cta(full + st, par, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t a = desc0 + st * stage_step, b = a + (W_TILE >> 4);
#pragma unroll
                for (int k = 0; k < 4; k++) umma_ss_by(lead, d, a + 2 * k, b + 2 * k, idesc, k || kb % KC);
                umma_commit_by(lead, empty + st);
                last = (int)(st * 2 + par);
                if (++st == (uint32_t)p.stages) { st = 0; par ^= 1; }
                if (kb % KC == KC - 1) {
                    umma_commit_by(lead, d_full + db);
                    if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
                }
            }
        }
        if (word_set(dead) && last >= 0) wait_flight(empty + (last >> 1), last & 1);      // given up: the products in flight
    } else if (warp >= EPI_WARP) {
        // ---- epilogue: a lane is a row of W; two warps share a quarter's rows, every other 16 tokens to each ----
        const int quarter = warp & 3, half = (warp - EPI_WARP) >> 2, r = quarter * 32 + lane;
        const uint32_t tq = ((uint32_t)(quarter * 32) << 16) + half * 16;
        uint32_t db = 0, dpar = 0;
        Place q = start(p, u0);
        pdl_wait();
        const float* token_scale = p.scale ? behind_wait(p.scale) : nullptr;
        for (int u = u0; u < u1;) {
            const int seg0 = u, end = min(u1, u + (p.NB - q.b));
            constexpr int G = PARTS == 3 ? (NT_FINE + 31) / 32 : NT_MAX / 32;
            uint64_t acc[G][8] = {}, unit[PARTS == 3 ? G : 1][8] = {};      // pairs of tokens; fine: a unit's first, which keeps the sums that small ones are added to small
            const uint64_t one = pack2(1.0f, 1.0f);
#pragma unroll 1
            for (int c = (end - u) * (4 / KC); c > 0; c--) {
                wait_cta(d_full + db, dpar, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int i = 0; i < G; i++) {
                    if (32 * i + 16 * half >= NT) break;
                    uint32_t v[PARTS][16];
#pragma unroll
                    for (int n = 0; n < PARTS; n++) tmem_ld16(tq + (db * PARTS + n) * NT + 32 * i, v[n]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 8; j++) {                  // what the parts gave first, the small ones first
                        uint64_t sum = pack2(__uint_as_float(v[PARTS - 1][2 * j]), __uint_as_float(v[PARTS - 1][2 * j + 1]));
#pragma unroll
                        for (int n = PARTS - 2; n >= 0; n--) sum = fma2(sum, one, pack2(__uint_as_float(v[n][2 * j]), __uint_as_float(v[n][2 * j + 1])));
                        if (PARTS == 2) acc[i][j] = fma2(sum, one, acc[i][j]);
                        else unit[i][j] = fma2(sum, one, unit[i][j]);
                    }
                }
                if (PARTS == 3 && c % 4 == 1)
#pragma unroll
                    for (int i = 0; i < G; i++)
#pragma unroll
                        for (int j = 0; j < 8; j++) { acc[i][j] = fma2(unit[i][j], one, acc[i][j]); unit[i][j] = 0; }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty + db);
                if (++db == (uint32_t)p.d_bufs) { db = 0; dpar ^= 1; }
            }
            u = end;
            finish_tile<G, 32>(p, q, acc, u0, seg0, end, 16 * half, r, token_scale, &last_smem, dead);
            q.b = 0; q.tile++;
            place(p, q);
        }
        if (word_set(dead)) report(p.status);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_smem), "n"(512));
}

template <int PARTS>
void launch_dense(const DenseMaps& maps, const DenseParams& p, int grid, cudaStream_t s) {
    static unsigned long long configured = 0;      // bit per device id
    opt_in_dynamic_smem(gemm_dense_tc_kernel<PARTS>, (int)SMEM_CAP + 1024, configured);
    launch_k_pdl(true, gemm_dense_tc_kernel<PARTS>, dim3(grid), dim3(THREADS), (size_t)p.stages * p.stage + 1024, s, maps, p);
    count_launch();
}

}  // namespace

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}
size_t dense_count_bytes() { return (size_t)sm_count() * sizeof(unsigned); }

// Times in us that the two were measured to take (1024 to 8192 rows, 1024 to 14336 columns, 32 to 1536 tokens; with either's split of the tokens): here tiles are spread over all SMs
// at 0.35 + 0.0025 NT for a k-block (HBM, then L2) and a tail for the tiles' shares; there a wave of tiles of 128 x 256 takes 0.78 for a k-block, however few they are.  4096 x 4096:
// 100 tokens 29 here, 54 there; 512 44, 52; 1024 73, 58.  2048 x 1024: 256 20, 22; 1024 27, 23.
bool gemm_dense_tc_pays(const int* N, int n, int T, int K, bool together) {
    const int sms = sm_count(), cols = (T + NT_MAX - 1) / NT_MAX, nt = ((T + cols - 1) / cols + 15) / 16 * 16;
    long long tiles = 0, waves = 0, wide = 0;
    for (int i = 0; i < n; i++) {
        tiles += (N[i] + 127) / 128 * (long long)cols;
        const int bn = !together && N[i] % 256 ? 128 : 256;
        const long long there = (N[i] + bn - 1) / bn * (long long)((T + 127) / 128);
        if (together) wide += there;
        else waves += (there + sms - 1) / sms;
    }
    if (together) waves = (wide + sms - 1) / sms;
    return (double)tiles / sms * (0.35 + 0.0025 * nt) * (K / 64) + 4.0 + 0.04 * nt < (double)waves * 0.78 * (K / 64);
}

bool gemm_dense_tc_supported(const GemvMat* mats, int n_mat, int K) {
    if (n_mat < 1 || n_mat > 3 || K <= 0 || K % 256) return false;
    for (int i = 0; i < n_mat; i++)
        if (mats[i].out < 1 || mats[i].dtype != mats[0].dtype || (mats[i].dtype != DType::F16 && mats[i].dtype != DType::BF16) || (mats[i].row_pitch && mats[i].row_pitch != (size_t)K * 2) ||
            (reinterpret_cast<uintptr_t>(mats[i].W) & 15)) return false;
    return true;
}

bool gemm_dense_tc(const GemvMat* mats, int n_mat, int K, const BlockTokens& x, void* scratch, int T, bool add, cudaStream_t s, const float* col_scale, float alpha) {
    if (T <= 0 || !gemm_dense_tc_supported(mats, n_mat, K)) return false;
    const int sms = sm_count();
    DenseParams p{};
    p.status = wait_status();
    p.n_mat = n_mat; p.T = T; p.NB = K / 256; p.add = add; p.bf16 = mats[0].dtype == DType::BF16;
    p.Mp = (T + 127) / 128 * 128;
    p.scale = x.scale; p.col_scale = col_scale; p.alpha = alpha;
    const int parts = x.fine ? 3 : 2;
    const int most = x.fine ? NT_FINE : NT_MAX;
    p.cols = (T + most - 1) / most;
    p.NT = ((T + p.cols - 1) / p.cols + 15) / 16 * 16;
    int tiles = 0;
    DenseMaps maps;
    if (!tc_map_f16(&maps.x, x.split, (uint64_t)parts * p.Mp, (uint64_t)K, (uint32_t)p.NT, p.bf16)) return false;
    for (int i = 0; i < n_mat; i++) {
        DealMat& m = p.mat[i];
        m.W = static_cast<const uint8_t*>(mats[i].W); m.C = mats[i].y; m.rows = mats[i].out; m.tiles = (m.rows + 127) / 128; m.pitch = (long long)K * 2;
        tiles += m.tiles;
        if (!tc_map_f16(&maps.w[i], m.W, (uint64_t)m.rows, (uint64_t)K, 128, p.bf16)) return false;
    }
    p.units = tiles * p.cols * p.NB;
    p.stage = W_TILE + parts * p.NT * 128;
    p.stages = std::min<int>(STAGES_MAX, (int)(SMEM_CAP / p.stage));
    p.d_bufs = std::min(BUFS_MAX, 512 / (parts * p.NT));
    p.part = static_cast<float*>(scratch);
    p.count = x.count;
    // whoever comes last reads the shares of a tile alone: no more of them than it reads in some 5 us (1024 x 4096, 100 tokens: 16 shares of 57 KB 54 us, 6 of
    // them 28)
    const int grid = std::min({sms, p.units, tiles * p.cols * std::max(4, 640 / p.NT)});
    if (parts == 3) launch_dense<3>(maps, p, grid, s);
    else launch_dense<2>(maps, p, grid, s);
    return true;
}

bool gemm_dense_tc(const GemvMat* mats, int n_mat, int K, const float* x, const float* norm_w, float eps, bool fine, int T, bool add, cudaStream_t s, const float* col_scale, float alpha) {
    if (T <= 0 || !gemm_dense_tc_supported(mats, n_mat, K) || (reinterpret_cast<uintptr_t>(x) & 15)) return false;
    const size_t scratch = block_scratch_bytes(NT_MAX);
    auto front = [&](int tokens) { return (block_tokens_bytes(tokens, K, fine) + 255) / 256 * 256; };
    int portion = (T + 127) / 128 * 128;
    for (int n = 2; portion > 128 && front(portion) + scratch > CALL_MEMORY_KEPT; n++) portion = ((T + n - 1) / n + 127) / 128 * 128;
    portion = std::min(portion, T);
    CallMemory memory(front(portion) + scratch, s);
    if (!memory.p) return false;
    GemvMat m[3];
    for (int t0 = 0; t0 < T; t0 += portion) {
        const int n = std::min(portion, T - t0);
        for (int i = 0; i < n_mat; i++) { m[i] = mats[i]; m[i].y += (size_t)t0 * mats[i].out; }
        const BlockTokens t = split_tokens(memory.p, x + (size_t)t0 * K, norm_w, eps, n, K, fine, s, mats[0].dtype == DType::BF16 ? TokenParts::BF16 : fine ? TokenParts::F16_SHORT : TokenParts::F16);
        if (!gemm_dense_tc(m, n_mat, K, t, static_cast<uint8_t*>(memory.p) + front(portion), n, add, s, col_scale, alpha)) return false;
    }
    return true;
}

}}  // namespace nt::b200
