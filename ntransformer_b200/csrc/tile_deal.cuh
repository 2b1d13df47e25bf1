// tile_deal.cuh — the dealing out of work in the GEMMs whose tiles are 128 rows of weights times some tokens (prefill_blocks.cu, prefill_dense.cu), and the end of a tile.
//
// Work is tiles times units of 256 columns, dealt out evenly: a CTA takes a run of units, whichever tiles it touches.  A tile that several CTAs share goes to a scratch, and whoever
// comes last adds the shares in their order: nothing waits for another CTA, and the sums do not depend on who was last.
#pragma once
#include "ring.cuh"
#include "wait_status.cuh"
#include "gemv_mma_device.cuh"

namespace nt { namespace b200 {
namespace {

struct DealMat { const uint8_t* W; float* C; int rows, tiles, fmt; long long pitch; };
struct Deal {
    DealMat mat[3];
    int n_mat, T, NT, cols, NB, add;      // tokens, of a tile, tiles of them, units of a row
    int units;                 // tiles * NB
    const float* scale;        // of a token's products; null: 1
    const float* col_scale;    // of a row's; null: 1
    float alpha;               // of all
    float* part;               // two tiles to a CTA
    unsigned* count;           // one to a CTA: shares of its last tile that have arrived; zeros at first
};
constexpr int EPI_WARP = 4;    // the first of the eight warps that take the sums

__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

// Where a CTA's run of units (tile * NB + super-block) stands; tokens inside, so that the CTAs of a wave share rows
struct Place { int tile, b, mi, row0, t0; };
__device__ __forceinline__ int first_unit(const Deal& p, int cta) { return (int)((long long)p.units * cta / (int)gridDim.x); }
__device__ __forceinline__ void place(const Deal& p, Place& q) {
    const int rt = q.tile / p.cols;
    q.t0 = (q.tile - rt * p.cols) * p.NT;
    int r = rt, mi = 0;
    if (p.n_mat > 1 && r >= p.mat[0].tiles) { r -= p.mat[0].tiles; mi = 1; }
    if (p.n_mat > 2 && mi == 1 && r >= p.mat[1].tiles) { r -= p.mat[1].tiles; mi = 2; }
    q.mi = mi; q.row0 = r * 128;
}
__device__ __forceinline__ Place start(const Deal& p, int u0) { Place q; q.tile = u0 / p.NB; q.b = u0 - q.tile * p.NB; place(p, q); return q; }
__device__ __forceinline__ void next(const Deal& p, Place& q) { if (++q.b == p.NB) { q.b = 0; q.tile++; place(p, q); } }

// The epilogue's end of a tile: this CTA's sums of units [seg0, end), 16 tokens of every STEP from `from` on.  A tile that other CTAs have a share of goes to the scratch, and
// whoever comes last adds the shares in their order.  named barrier 5: the epilogue's threads, two warps to a row where STEP is 32.
template <int N, int STEP>
__device__ __forceinline__ void finish_tile(const Deal& p, const Place& q, uint64_t (&acc)[N][8], int u0, int seg0, int end, int from, int r, const float* token_scale, uint32_t* last_smem, uint32_t dead) {
    const int NT = p.NT, live = min(NT, p.T - q.t0), rows = p.mat[q.mi].rows, row = q.row0 + r;
    bool write = true;
    if (end - seg0 < p.NB) {                                       // shared: to the scratch; whoever comes last adds
        write = false;
        const int tu = q.tile * p.NB, G = gridDim.x;
        const int c0 = (int)(((long long)(tu + 1) * G - 1) / p.units), c1 = (int)(((long long)(tu + p.NB) * G - 1) / p.units);
        float* mine = p.part + (size_t)(2 * blockIdx.x + (seg0 == u0 ? 0 : 1)) * 128 * NT + r;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int n = STEP * i + from;
            if (n >= live) break;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float x, y;
                unpack2(acc[i][j], x, y);
                __stcg(mine + (n + 2 * j) * 128, x);
                __stcg(mine + (n + 2 * j + 1) * 128, y);
            }
        }
        __threadfence();
        named_sync<8 * STEP>(5);
        if (threadIdx.x == EPI_WARP * 32) {
            const bool alive = !word_set(dead);
            const bool is_last = alive && atomicAdd(p.count + c0, 1u) == (unsigned)(c1 - c0);
            if (is_last) p.count[c0] = 0;
            __threadfence();
            *last_smem = is_last;
        }
        named_sync<8 * STEP>(5);
        if (*last_smem) {
            write = true;
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = 0;
#pragma unroll 1
            for (int c = c0; c <= c1; c++) {
                const float* o = p.part + (size_t)(2 * c + (first_unit(p, c) >= tu ? 0 : 1)) * 128 * NT + r;
#pragma unroll
                for (int i = 0; i < N; i++) {
                    const int n = STEP * i + from;
                    if (n >= live) break;
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = __ldcg(o + (n + j) * 128);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        float x, y;
                        unpack2(acc[i][j], x, y);
                        acc[i][j] = pack2(x + v[2 * j], y + v[2 * j + 1]);
                    }
                }
            }
        }
    }
    if (write && row < rows && !word_set(dead)) {                  // a warp stores 128 contiguous bytes for each token
        float* o = p.mat[q.mi].C + (size_t)(q.t0 + from) * rows + row;
        const float g = p.col_scale ? p.alpha * p.col_scale[row] : p.alpha;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int n = STEP * i + from;
            if (n >= live) break;
            float4 ts[4];                                          // (one by one between the stores they were a trip to L2 each: 9500 cycles for 64 tokens)
#pragma unroll
            for (int j = 0; j < 4; j++) ts[j] = token_scale ? __ldg(reinterpret_cast<const float4*>(token_scale + q.t0 + n) + j) : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                float x, y;
                unpack2(acc[i][j >> 1], x, y);
                const float4 s = ts[j >> 2];
                const float v = ((j & 1) ? y : x) * ((j & 3) == 0 ? s.x : (j & 3) == 1 ? s.y : (j & 3) == 2 ? s.z : s.w) * g;
                // adds go to the memory's side (this lane is the element's only writer): nothing is waited for
                if (n + j < live) {
                    if (p.add) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(o + (size_t)j * rows), "f"(v) : "memory");
                    else o[(size_t)j * rows] = v;
                }
            }
            o += (size_t)STEP * rows;
        }
    }
}

}  // namespace
}}  // namespace nt::b200
