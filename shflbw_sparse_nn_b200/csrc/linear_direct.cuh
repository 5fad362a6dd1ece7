// A linear layer on a handful of tokens in one launch: out[M][N] = W . x^T + bias with x token-major, as it arrives.
// One block: one row block and 8 tokens.
//
// Bound by latency and launches: 37 tokens of a 4096 x 4096 layer at density 0.1 are 0.13 GFLOP and 4 MB.  Transposing x first so that the
// panel kernel can gather whole rows takes a second launch (2.2 us of host time, 1.7 us of device time) and a buffer.
// Here a block gathers the elements of its columns straight from the tokens' rows: 32 lanes read 32 consecutive columns of
// one token's list, which at density 0.1 lie in 20 sectors (16 columns each: nearly the whole row is fetched), past L1, which
// would see no sector twice.  So a block reads about its share of x once, and the tokens are split over the blocks that share
// a row block as far as the SMs reach.  What it has gathered is K-major, the order in which mma.sync takes its second operand;
// the value panels are in the byte order of ldmatrix.  mma.sync and not tcgen05: the products are a few hundred cycles,
// and neither TMEM nor its barriers are worth setting up.
// A warp adds up 16 rows' products in the order of the columns, 16 at a time, as the panel kernel does, and gets its bits.
// (Columns dealt out over all warps and their sums added: 1 % less time over 90 shapes.  256 columns a pass with the next two
// passes in flight: 8 % more.  16 to 32 tokens a block: 10 to 60 % more.)
#pragma once

#include <cstdint>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "shflbw_internal.hpp"
#include "sm100_ptx.cuh"

namespace shflbw {

constexpr int kDirectTokens = 8;                              // of a block: one n of mma.sync
constexpr int kDirectCols = 512;                              // columns of a block in shared memory at a time
constexpr int kDirectPitch = kDirectCols * 2 + 16;            // bytes of a token's gathered columns (eight tokens: 32 banks)

struct DirectParams {
    const int *blk_ptr, *blk_idx, *perm;
    const __half *blk_val, *x, *bias;
    __half* out;
    int tokens, K, N, groups;                                 // groups: blocks of 8 tokens that share a row block
};

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

inline size_t direct_smem(int V, int max_cols) {
    return kDirectTokens * kDirectPitch + (size_t)(max_cols < kDirectCols ? max_cols : kDirectCols) * V * 2;
}

template <int V>
__global__ void __launch_bounds__(256) linear_direct(const DirectParams p) {
    constexpr int RUNS = kDirectCols / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    sm100::grid_dependency_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int blk = blockIdx.x / p.groups, t0 = (blockIdx.x - blk * p.groups) * kDirectTokens;
    const int row0 = __ldg(p.blk_ptr + blk), cols = __ldg(p.blk_ptr + blk + 1) - row0;       // a multiple of 16
    unsigned char* const xs = smem;                           // the gathered columns, then the value panels
    const uint32_t w_smem = sm100::smem_u32(smem) + kDirectTokens * kDirectPitch;
    const bool mine = t0 + warp < p.tokens;                   // warp w gathers token w
    const unsigned short* const x = (const unsigned short*)p.x + (size_t)(mine ? t0 + warp : 0) * p.K;

    float acc[4] = {};                                        // warp w: rows 16 w to 16 w + 15 of the block
    int c0 = 0;
    do {
        const int n = cols - c0 < kDirectCols ? cols - c0 : kDirectCols;
        // The value panels and the column ids are the layer's own: requested before the previous kernel is waited for.  (Not a
        // word of arithmetic on the ids here: clamped as they are loaded, each load was waited for by itself, 4.9 us instead of
        // 2.95 at 256 x 840, V = 128, 26 tokens.)
        const __half* const w = p.blk_val + (size_t)(row0 + c0) * V;
        for (int i = tid; i < n * (V / 8); i += 256) sm100::cp_async_16(w_smem + i * 16, w + i * 8, 16);
        sm100::cp_async_commit();
        int id[RUNS];
#pragma unroll
        for (int s = 0; s < RUNS; ++s) id[s] = mine && s * 32 + lane < n ? __ldg(p.blk_idx + row0 + c0 + s * 32 + lane) : -1;
        if (c0 == 0) sm100::grid_dependency_wait();           // x may be the previous kernel's output
        unsigned short v[RUNS];                               // sixteen runs of 32 columns in flight
#pragma unroll
        for (int s = 0; s < RUNS; ++s)                        // (clamped: a corrupted id may give wrong numbers, never an address outside x)
            v[s] = id[s] >= 0 ? __ldcg(x + min(id[s], p.K - 1)) : (unsigned short)0;
#pragma unroll
        for (int s = 0; s < RUNS; ++s)
            *(unsigned short*)(xs + warp * kDirectPitch + (s * 32 + lane) * 2) = v[s];
        sm100::cp_async_wait<0>();
        __syncthreads();
        if (warp < V / 16) {
#pragma unroll 4
            for (int k = 0; k < n; k += 16) {
                const unsigned char* const src = xs + (lane >> 2) * kDirectPitch + (k + 2 * (lane & 3)) * 2;
                uint32_t a[4];                                // 8 x 8: rows 0-7 / 8-15 of columns 0-7, then of columns 8-15
                const int m = warp * 16 + ((lane >> 3) & 1) * 8, r = k + (lane >> 4) * 8 + (lane & 7);
                sm100::ldmatrix_x4_trans(w_smem + (uint32_t)kval_index(V, r, m) * 2, a);
                mma_16816(acc, a, *(const uint32_t*)src, *(const uint32_t*)(src + 16));
            }
        }
        __syncthreads();                                      // before this memory is written again
        c0 += kDirectCols;
    } while (c0 < cols);

    if (warp >= V / 16) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {                             // a lane: two tokens of rows l / 4 and l / 4 + 8; four lanes: 16 bytes
        const int m = blk * V + warp * 16 + (lane >> 2) + 8 * i;
        const int row = p.perm ? __ldg(p.perm + m) : m;
        __half2 y = __floats2half2_rn(acc[2 * i], acc[2 * i + 1]);
        if (p.bias) y = __hadd2(y, __half2half2(p.bias[row]));        // added to the fp16 product, as the panel kernel does
        *(__half2*)(p.out + (size_t)row * p.N + t0 + 2 * (lane & 3)) = y;   // t0 + 8 <= N, a multiple of 8
    }
}

}  // namespace shflbw
