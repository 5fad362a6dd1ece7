// The Shfl-BW panel kernel for sm_100a (persistent, warp-specialised).
//
// Work item = ONE row block of V stored rows x ONE tile of T = 128*TM dense columns
// ("tokens": SpMM columns of B, or SpConv output positions).  For an item the kernel
// computes the dense contraction
//
//     acc[token][m] = sum_p  G[p][token] * W[p][m]          p over the block's non-zero columns
//
// on the 5th-generation tensor cores, K = 16 per instruction, both operands MN-major in shared
// memory: W[p][0..V) is a contiguous slice of the value panels, G[p][..] is row indices[p] of
// the dense operand, gathered from L2.  Two orientations exist (template parameter MODE):
//   tokens in lanes  tokens are the UMMA M dimension (128 TMEM lanes), the V rows of the block
//                    the N dimension (16/32/64/128): TM instructions per 16 columns.  V = 16 and
//                    32, SpConv writing NHWC, and what the rules below keep from the other.
//   rows in lanes    the V rows are M (64 or 128) and the T tokens N (128 or 256): ONE instruction
//                    per 16 columns, 128 clk at 128 x 256, 80 clk at 64 x 256 (weight-stationary
//                    form), and the accumulator holds one output row per lane.  V = 64 / 128:
//                    SpMM by the layout of D, C and the depth (spmm_rows, spmm_wide), chained
//                    SpConv where it is deep (chain_rows), planes of very deep 64-row filters.
// The description below is written for the first orientation; the second differs in the
// gathered tile's layout ([K group][T/64 swizzle atoms]), the MMA issue and the epilogue.
//
// One CTA per SM loops over items (item = blockIdx.x + i*gridDim.x, decoded block-major or
// tile-major, PanelParams::tile_major); their extents are read once into a shared-memory table.
// Warp roles (warp w issues from scheduler partition w % 4; EW = 8 or 16 epilogue warps):
//   warps 0..EW-1    epilogue.  Warp w reads TMEM lane quadrant w % 4 and half w / 4 % 2 of the
//                    accumulator columns; sixteen warps are two sets that take the items in turn.  Tokens in lanes: TMEM -> registers -> fp16 -> transpose
//                    of 32-row chunks through shared memory -> 16-byte global stores (inverse row
//                    permutation fused for SpMM).  Rows in lanes: stores straight from registers.
//   warp  EW         allocates TMEM; an elected lane issues tcgen05.mma, releases stages and
//                    accumulators with tcgen05.commit
//   warps EW+1.. with w % 4 != 0   producers (PW of them, in GROUPS groups that take the stages in
//                    turn).  cp.async gather: 16-byte copies into 128-byte-swizzled stages; a
//                    group publishes its previous stage half-way through issuing the next one,
//                    with ONE mbarrier arrival per warp; row ids are prefetched two of the
//                    group's stages ahead by 4-byte cp.async into a shared-memory ring.  TMA
//                    gather (every warp after the MMA warp): tile::gather4 copies, completion by byte count.
//                    One bulk copy per stage for the value slice either way.
//   later warps with w % 4 == 0   beside cp.async producers idle, so that none shares the MMA warp's scheduler partition.
// The accumulator is double buffered in TMEM (four sets with EW = 16 and with 64 rows in lanes) so the epilogue of item i
// overlaps the main loop of item i+1, and the stage ring runs across item boundaries without
// draining.
//
// Every mbarrier wait is bounded (sm100_ptx.cuh): on a timeout the kernel records a code in
// the status word, raises a CTA-wide abort flag, drains and exits; it cannot hang the GPU.
//
// Replaces SpmmBlockwiseKernel::mainLoop / epilogue (block_sparse/spmm/blockwise_kernel.h:99-294,
// block_sparse/common/epilogue.h:6-135) and SpconvBlockwiseKernel::mainLoop
// (block_sparse/spconv/blockwise_kernel.h:63-261, block_sparse/spconv/conv_format.h:14-82).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "shflbw.h"
#include "sm100_ptx.cuh"

namespace shflbw {

constexpr long long kWaitLimitCycles = 400000000LL;   // default bound of every in-kernel wait: ~0.2 s at 2 GHz

// Division of a non-negative int below 2^31 by a divisor fixed per launch: the quotient is
// umulhi(n, mul) >> shr with mul = ceil(2^(31 + ceil(log2 d)) / d), shr = ceil(log2 d) - 1
// (d == 1: the number itself).  Four instructions instead of the ~25 of a 32-bit division in
// software; the epilogues of shallow items are instruction-bound and divide three times per item.
struct FastDiv {
    unsigned d, mul, shr;
};
inline FastDiv make_fast_div(int d) {
    FastDiv f{(unsigned)d, 0u, 0u};
    if (d > 1) {
        const unsigned c = 32 - __builtin_clz((unsigned)d - 1);  // ceil(log2 d)
        const unsigned p = 31 + c;
        f.mul = (unsigned)(((1ull << p) + (unsigned long long)d - 1) / (unsigned long long)d);
        f.shr = p - 32;
    }
    return f;
}
__device__ __forceinline__ int fast_div(int n, const FastDiv& f) {
    return f.d == 1u ? n : (int)(__umulhi((unsigned)n, f.mul) >> f.shr);
}

struct alignas(64) PanelParams {
    // TMA gather only: tensor map of the dense operand (SpMM: B[K][N]; SpConv: one row per pixel of the staged
    // input, running from that pixel to the end of what a tap reads; box = 64 tokens x 1 row, 128-byte swizzle);
    // first member so that it sits on the 64-byte boundary the copy engine wants
    unsigned long long tmap_b[16];
    unsigned long long tmap_res[16];   // box epilogue only: tensor map of the residual's planes (box = 64 tokens x 1 plane)
    // sparse operand (kernel image)
    const int* blk_ptr;      // [X+1] padded offsets (multiples of 16)
    const int* blk_idx;      // padded column ids
    const __half* blk_val;   // value panels of the padded rows, element order kval_index() (shflbw_internal.hpp)
    const int* perm;         // [M] or nullptr
    int* status_word;
    unsigned idx_limit;      // cp.async gather: largest legal offset, K - 1 (SpMM, a row id) or the element offset of the
                             // last (channel, tap) plane origin (SpConv).  Ids are clamped to it, so a corrupted id can
                             // give wrong numbers but never an address outside the dense operand; the TMA gather reads
                             // zeros for a row that its map does not have
    long long wait_limit;    // SM clocks after which a barrier wait gives up (kWaitLimitCycles unless the host overrides it)
    float alpha, beta;
    int num_items, tiles_n;  // work items = row blocks x token tiles; item -> (item / tiles_n, item % tiles_n)
    FastDiv div_tiles, div_bp, div_row;  // division by tiles_n, Bp, row_pix (set by the host with make_fast_div)
    // Order of the work items.  0: item = block * tiles_n + tile (a CTA's neighbours work on the
    // same row block).  1: item = tile * num_blocks + block: the CTAs that run at the same time
    // share a few token tiles, so the rows of the dense operand they gather are a small set that
    // stays in L2 (SpMM with a large dense operand).
    int tile_major, num_blocks;
    FastDiv div_blocks;
    int inject_from;         // fault-injection builds only (-DSHFLBW_FAULT_INJECT): from this stage number on, one
                             // producer warp withholds its arrivals, so the consumer's bounded wait runs out (< 0: off)
    // SpMM
    const __half* B;         // [K][N]
    const __half* C;         // [M][N] or nullptr; kernels built with BIAS: one value per output row / filter
    __half* D;               // [M][N]
    int N;                   // dense columns (SpMM) / Ho*row_pix*Bp (SpConv)
    // SpConv (input staged channel-major, batch innermost, with a zero halo:
    // Xs[c][Hp][Wp][Bp], Hp = Hin + R - 1, Wp = Win + S - 1, image origin at (R/2, S/2); a strided 1x1
    // filter of an NHWC call is staged as the pixels it visits, Hp = Ho, Wp = Wo, and read at stride 1)
    const __half* Xs;
    __half* out;             // [B*Ho*Wo][F] (NHWC) -- final or staged in stored filter order
    int Bn, Bp, Hp, Wp, Cin, F, R, S, stride, Ho, Wo;
    // An output row counts as row_pix >= Wo pixels: with the TMA gather a row may be rounded up so that no box of 64
    // tokens crosses from one into the next, where the input's halo makes addresses jump.  Tokens of pixels
    // ow >= Wo are computed from whatever is there and stored nowhere.
    int row_pix;
    // chained SpConv: out[f][OHp][OWp][Bp] with the next layer's halo (origin at (oph, opw))
    int OWp, oph, opw, out_plane, relu;
    int wide_stores;         // SpMM, rows in lanes: output rows are 32-byte aligned (N % 16 == 0, D % 32 == 0)
    int trigger_late;        // SpConv ending with this kernel (nothing left to permute): lets its dependents in when its producers are done
    int out_logical;         // chained kernels: output plane of stored filter f is perm[f] (logical channel order) instead of f
    const __half* res;       // optional residual in the OUTPUT's geometry ([planes][OHp][OWp][Bp]) or nullptr
    const int* res_map;      // stored filter -> plane of `res` (nullptr: same index)
};

// MODE: 0 = SpMM, 1 = SpConv writing NHWC (stored filter order), 2 = SpConv writing the
// channel-major halo layout the next layer gathers from ("chained" layers).
// 3 = SpMM with the operands swapped: the block's V rows are the UMMA M dimension (64 or 128
// TMEM lanes) and the T tokens the N dimension, so ONE instruction per 16 columns covers the
// whole token tile and the accumulator comes out with an output row per lane.
// 4 = chained SpConv with the operands swapped in the same way.
// 5 = SpConv writing NHWC in logical filter order, value by value (a kernel of its own: as a branch of 1 it cost that 1 to 3 %).
constexpr int kPanelSpmm = 0, kPanelConv = 1, kPanelConvChain = 2, kPanelSpmmRows = 3, kPanelConvChainRows = 4,
              kPanelConvScatter = 5;

// GATHER: how the rows of the dense operand reach shared memory.
//   kGatherCpAsync  16-byte cp.async per lane, written straight into the swizzled layout; the
//                   producer warps wait for their copies and publish the stage themselves.
//   kGatherTma      TMA tile::gather4: one instruction fetches 4 rows x 64 tokens (the tensor map covers
//                   this GPU's own dense operand; no multicast), the copy engine applies the 128-byte
//                   swizzle and completes the stage's barrier by byte count, so the producers never
//                   wait for data.
constexpr int kGatherCpAsync = 0, kGatherTma = 1;

// EW: epilogue warps, 8 or 16.  A warp can read only the TMEM lane quadrant warp % 4, so the two
// warps of a quadrant split the accumulator columns between them.  Items with few non-zero
// columns are all epilogue, and one warp's chain (TMEM read, convert, transpose, store) is
// latency-bound: sixteen warps, as two sets on alternate items, keep four such chains per
// scheduler in flight instead of two.
template <int V, int TM, int KS_, int STAGES, int PW, int MODE, int GROUPS_ = 2, int GATHER_ = kGatherCpAsync,
          int EW_ = 8, bool ADDEND_ = false, int SLOTS_ = 0>
struct PanelCfg {
    static constexpr int EW = EW_;
    static_assert(EW == 8 || EW == 16, "epilogue warps");
    static constexpr bool TMA = GATHER_ == kGatherTma;
    static constexpr int KS = KS_;                         // non-zero columns per pipeline stage
    static constexpr int T = 128 * TM;
    static constexpr int GROUPS = GROUPS_;                 // producer groups that take the stages in turn
    // Warp w runs on scheduler partition w % 4.  The MMA warp (the first after the epilogue
    // warps: 8 or 16) sits on partition 0; beside cp.async producers the later warps with
    // w % 4 == 0 stay idle: the MMA thread executes a few dozen instructions per stage and was
    // measured at ~20 clk per instruction when their code kept evicting its lines from the
    // partition's instruction cache.
    static constexpr int WARPS = EW + 1 + PW + (TMA ? 0 : (PW - 1) / 3);   // epilogue + MMA + producers + idle
    static_assert(EW == 8 || WARPS <= 20, "16 epilogue warps: at most 3 producers (20 warps leave 96 registers per thread, 21-24 only 80)");
    static constexpr int THREADS = WARPS * 32;
    static constexpr int G_ACC = KS * 256;                 // gathered tile of one accumulator: [KS][128] fp16
    static constexpr int G_BYTES = TM * G_ACC;
    static constexpr int W_BYTES = KS * V * 2;
    static constexpr int STAGE_BYTES = G_BYTES + W_BYTES;
    static constexpr int PIPE_BYTES = STAGES * STAGE_BYTES;
    // Epilogue tiles (tokens in lanes only): each epilogue warp transposes 32 tokens x 32 output
    // rows / filters through 2 KB so that its global stores are 16 bytes per lane and 64-byte
    // runs.  With rows in lanes the stores go straight from registers.
    // Box epilogue: SLOTS slots of 32 rows x 64 tokens per pair of warps.
    static constexpr int SLOTS = SLOTS_, SLOT_ROWS = 32, SLOT_BYTES = SLOT_ROWS * 128;
    static constexpr int OUT_BYTES = (MODE == kPanelSpmmRows || MODE == kPanelConvChainRows) ? 0 : SLOTS ? EW / 2 * SLOTS * SLOT_BYTES : EW * 2048;
    // Sixteen epilogue warps, instances built with ADDEND: the addend of an item (C, or a chained layer's
    // residual) is copied to shared memory an item ahead: each lane's own 16-byte pieces, 64 rows x 32
    // tokens per warp.  Without, the ring has that room.
    static_assert(!ADDEND_ || EW == 16, "addend slots: sixteen epilogue warps");
    static constexpr int RES_BYTES = ADDEND_ ? EW * 4096 : SLOTS ? EW * SLOT_ROWS * 4 : 0;   // (box epilogue: row ids of a refill)
    static constexpr int SLOT_BARS = SLOTS ? EW / 2 * (SLOTS + 1) : 0;       // per pair: one for each slot, one for its two warps
    static constexpr int BAR_BYTES = (STAGES * 2 + 12 + SLOT_BARS) * 8;  // mbarriers (ring, up to 4 + 4 accumulator, drain) + tmem slot + abort flag
    static constexpr int TAB_BYTES = 512 * 8;               // per-CTA item table (kPanelMaxItemsPerCta entries)
    static constexpr int IDX_AHEAD = 2;                    // a group fetches row ids this many of its stages ahead
    static constexpr int IDX_RING = (IDX_AHEAD + 1) * GROUPS <= 8 ? 8 : 16;   // stages of row ids kept in shared memory
    static_assert((IDX_AHEAD + 1) * GROUPS <= IDX_RING, "row-id ring too small");
    static constexpr int IDX_BYTES = (TMA ? PW : IDX_RING) * KS * 4;     // (TMA gather: one stage of row ids per producer warp)
    static constexpr int SMEM_BYTES = PIPE_BYTES + OUT_BYTES + RES_BYTES + BAR_BYTES + TAB_BYTES + IDX_BYTES + 1024;  // + align slack
    static constexpr bool SWAP = MODE == kPanelSpmmRows || MODE == kPanelConvChainRows;
    static constexpr int KG_BYTES = SWAP ? T * 16 : 2048;   // 8 gathered rows (one K group) of the token tile
    // 64 rows in lanes run as weight-stationary MMAs (tcgen05.mma.ws): 80 clk for 64 x 256 x 16 instead of 128, and
    // the accumulator fills all lanes: token t of row m is lane m + 64 * (t / (T / 2)), column t % (T / 2).
    static constexpr bool WS = SWAP && V == 64;
    static constexpr uint32_t ACC_COLS = WS ? T / 2 : SWAP ? T : TM * V; // fp32 columns of one accumulator set
    static_assert(!SWAP || V == 64 || V == 128, "rows-in-lanes needs a legal UMMA M");
    // Accumulator sets in TMEM: two (the MMAs of item i+1 run while the epilogue reads item i);
    // four with sixteen epilogue warps, whose items are so short that the hand-over itself
    // (commit -> barrier -> poll -> TMEM read -> release -> poll -> issue) is what two sets
    // cannot hide.
    // Sixteen epilogue warps work as two sets of eight that take the items in turn, so that the chains
    // of two items (accumulator wait, TMEM read, transpose, stores) overlap.
    static constexpr int ESETS = EW / 8;
    static constexpr int NBUF = ((EW == 16 || WS) && ACC_COLS * 4 <= 512) ? 4 : 2;
    static constexpr uint32_t TMEM_COLS = NBUF * ACC_COLS < 32 ? 32 : NBUF * ACC_COLS;
    static_assert(V == 16 || V == 32 || V == 64 || V == 128, "row-block height");
    static_assert(V != 16 || !SWAP, "16-row blocks: tokens in lanes");
    static_assert(!TMA || (GROUPS <= STAGES && (KS / 4) % (PW / GROUPS) == 0), "TMA gather: producer groups, row quads per warp");
    static_assert(STAGE_BYTES % 1024 == 0, "stages must keep 1024-byte swizzle-atom alignment");
    static_assert((TMEM_COLS & (TMEM_COLS - 1)) == 0 && TMEM_COLS <= 512, "TMEM columns");
    static_assert(KS % 32 == 0 && PW % GROUPS == 0 && (TMA || (KS % (PW / GROUPS) == 0 && (KS / (PW / GROUPS)) % (32 / (T / 8)) == 0)),
                  "rows per producer warp");
    static_assert(TMA || STAGES > GROUPS, "a group publishes a stage while issuing its next one");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

// Shared-memory tile layouts (MN-major operands; r = K row inside the stage, c = 16-byte
// chunk along MN).  A 128-byte-swizzle atom is 8 K rows x 128 bytes (64 fp16 along MN); the
// chunk index inside a row is XORed with r % 8.
//   two atoms wide (128 fp16 along MN):  K group g = r / 8 at g*2048, MN atom c / 8 at +1024
//       -> descriptor LBO = 1024 (next MN atom), SBO = 2048 (next K group); K-step j at j*4096
//   one atom wide (64 fp16):             K group at g*1024 -> SBO = 1024; K-step j at j*2048
//   64-byte swizzle, 32 fp16 wide:       atom = 8 rows x 64 bytes, chunk XOR (r/2)%4,
//                                        K group at g*512 -> SBO = 512; K-step j at j*1024
__device__ __forceinline__ uint32_t tile128_off(int r, int c) {
    return (uint32_t)((r >> 3) * 2048 + (c >> 3) * 1024 + (r & 7) * 128 + (((c & 7) ^ (r & 7)) << 4));
}
__device__ __forceinline__ uint32_t tile64_off(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }
__device__ __forceinline__ uint32_t tile32_off(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }

// The value at p in all eight halves of 16 bytes.
__device__ __forceinline__ uint4 broadcast8(const __half* p) {
    const uint32_t h = __ldg((const unsigned short*)p) * 0x10001u;
    return make_uint4(h, h, h, h);
}

constexpr int kPanelMaxItemsPerCta = 512;  // capacity of the per-CTA item table

// Epilogue of a chained layer with a residual that comes in boxes (64 consecutive tokens are 128 consecutive bytes of a
// plane; tokens in lanes).  Such a layer is all epilogue, and what bounded it was the load/store unit: 2 250 wavefronts an
// item of 64 x 256, 1 200 of them the residual's cp.async in 64-byte pieces.  Here the copy engine fetches the residual,
// by tile::gather4 (its planes are permuted), into slots [row][64 tokens], 128-byte-swizzled.  The accumulator comes
// out of TMEM as 8 x 8 tiles, is added to the residual in that form (ldmatrix transposes), goes back into the slot
// (stmatrix) and leaves as 16-byte pieces of rows.  (Stores by TMA, a box at a time, were slower: 8 clk of the engine for
// 128 bytes.)
//
// A pair of warps (TMEM quadrants 2 j and 2 j + 1, the same columns) shares a box and SLOTS slots, which its chunks of
// 32 rows take in turn.  When warp q % 2 has finished chunk q + 1, and the other warp chunk q, it has chunk q's slot
// refilled for chunk q + SLOTS.  All waits are on mbarriers and bounded.
template <class Cfg, int V, class ItemBlock, class ItemTile>
__device__ __forceinline__ void box_epilogue(const PanelParams& p, uint8_t* smem, uint32_t smem_base, uint32_t tmem_base, const int2* item_tab, int nloc,
                                             uint64_t* acc_full, uint64_t* acc_empty, uint64_t* slot_bar, volatile int* cta_abort,
                                             int warp, int lane, const ItemBlock& item_block, const ItemTile& item_tile) {
    constexpr int NBUF = Cfg::NBUF, ESETS = Cfg::ESETS, T = Cfg::T, NS = Cfg::SLOTS, ROWS = Cfg::SLOT_ROWS, D = NS - 1;
    constexpr int COLS = Cfg::ACC_COLS / 2, NCH = COLS / ROWS;
    static_assert(NCH * ROWS == COLS && COLS <= V, "chunks of one accumulator");
    static_assert(NS >= 2, "a chunk is added to while the one before is on its way out");
    const int quad = warp & 3, half_id = (warp >> 2) & 1, first = ESETS > 1 ? warp >> 3 : 0;
    const int a0 = half_id * COLS / V, mbase = half_id * COLS % V;     // accumulator and first block row of this warp
    const int pair = first * 4 + half_id * 2 + (quad >> 1), me = quad & 1;
    uint64_t* const ready = slot_bar + pair * NS;              // [NS] residual landed
    uint64_t* const done = slot_bar + Cfg::EW / 2 * NS + pair;         // the warp that does not refill the slot is done with it
    const uint32_t slots = smem_base + (uint32_t)(Cfg::PIPE_BYTES + pair * NS * Cfg::SLOT_BYTES);
    int4* const ids = (int4*)(smem + Cfg::PIPE_BYTES + Cfg::OUT_BYTES + warp * (ROWS * 4));   // planes of the next refill
    // stmatrix: lane 8 k + j names tokens 8 k.. of this warp's 32, row 8 i + j; the 16-byte chunk is XORed with j.  Pieces:
    // lane 4 j + c takes tokens 8 c.., row 8 i + prow: rows r and r + 4 in turn, so that eight lanes read all banks.
    const uint32_t lane_off = (uint32_t)((lane & 7) * 128 + (((me * 4 + (lane >> 3)) ^ (lane & 7)) << 4));
    const int prow = ((lane >> 2) & 1) * 4 + (lane >> 3);
    const uint32_t piece_off = (uint32_t)(prow * 128 + (((me * 4 + (lane & 3)) ^ prow) << 4));
    const __half2 alpha2 = __half2half2(__float2half_rn(p.alpha)), zero2 = __float2half2_rn(0.f);
    if (warp == 0 && sm100::elect_one()) sm100::prefetch_tensormap(p.tmap_res);
    auto offset = [&](int tok) {                               // of a token's element in a plane
        const int pix = fast_div(tok, p.div_bp), oh = fast_div(pix, p.div_row);
        return ((oh + p.oph) * p.OWp + pix - oh * p.row_pix + p.opw) * p.Bp + tok - pix * p.Bp;
    };
    auto first_tok = [&](int item) { return item_tile(item) * T + a0 * 128 + (quad >> 1) * 64; };   // of the pair's box
    auto load_ids = [&](int li, int ch) {                      // planes of four rows per lane, lanes 0..ROWS/4-1
        const int f = item_block((int)blockIdx.x + li * (int)gridDim.x) * V + mbase + ch * ROWS + lane * 4;
        return lane >= ROWS / 4 || li >= nloc ? make_int4(0, 0, 0, 0) : p.res_map ? __ldg((const int4*)(p.res_map + f)) : make_int4(f, f + 1, f + 2, f + 3);
    };
    auto refill = [&](int li, const int4& id, uint32_t slot) { // by one warp of the pair
        const int tok = first_tok((int)blockIdx.x + li * (int)gridDim.x);
        if (lane < ROWS / 4) ids[lane] = id;
        __syncwarp();
        if (sm100::elect_one()) {
            if (tok < p.N) {
                const int x = offset(tok);
                int4 r[ROWS / 4];
#pragma unroll
                for (int i = 0; i < ROWS / 4; ++i) r[i] = ids[i];
                sm100::mbar_arrive_expect_tx(&ready[slot], (uint32_t)Cfg::SLOT_BYTES);
#pragma unroll
                for (int i = 0; i < ROWS / 4; ++i)
                    sm100::tma_gather4(slots + slot * (uint32_t)Cfg::SLOT_BYTES + (uint32_t)(i * 512), p.tmap_res, x, r[i].x, r[i].y, r[i].z, r[i].w, &ready[slot]);
            } else {
                sm100::mbar_arrive(&ready[slot]);
            }
        }
        __syncwarp();
    };
#pragma unroll
    for (int q = 0; q < NS; ++q)
        if (first + q / NCH * ESETS < nloc && (q & 1) == me) refill(first + q / NCH * ESETS, load_ids(first + q / NCH * ESETS, q % NCH), (uint32_t)q);
    uint32_t slot = 0, par = 0, q = 0, prev = 0;               // slot of chunk q, its parity; slot of chunk q - 1
    for (int li = first; li < nloc; li += ESETS) {
        const int item = (int)blockIdx.x + li * (int)gridDim.x, b = li % NBUF;
        const bool has_k = item_tab[li].y > 0;
        const int tok = first_tok(item) + me * 32 + (lane & 3) * 8;        // this lane's 8 tokens
        const bool ok = tok < p.N;
        __half* const dst = p.out + offset(tok);
        const int f0 = item_block(item) * V + mbase;
        const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + b * Cfg::ACC_COLS + half_id * COLS;
        if (!sm100::mbar_wait_warp(&acc_full[b], (li / NBUF) & 1, cta_abort, p.status_word, SHFLBW_DEVSTAT_TIMEOUT_ACCUM, p.wait_limit)) return;
        sm100::tc_fence_after_sync();
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
            const bool refills = (int)(q & 1) != me && q > 0;  // chunk q - 1's slot
            const int li_n = li + (ch + D) / NCH * ESETS;
            int4 id = make_int4(0, 0, 0, 0);
            if (refills) id = load_ids(li_n, (ch + D) % NCH);
            __half2 h[ROWS / 8][4];                            // tile of rows 8 i.., tokens 8 k..
            {
                uint32_t lo[ROWS / 2], hi[ROWS / 2];           // lanes 0-15 and 16-31 of the quadrant
                if (has_k) {
                    sm100::tmem_ld_16x256b(acc + ch * ROWS, lo);
                    sm100::tmem_ld_16x256b(acc + (16u << 16) + ch * ROWS, hi);
                    sm100::tmem_ld_wait();
                } else {
#pragma unroll
                    for (int e = 0; e < ROWS / 2; ++e) lo[e] = hi[e] = 0u;
                }
                if (ch + 1 == NCH) {                           // last TMEM read of this item by this warp: release the buffer
                    sm100::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) sm100::mbar_arrive(&acc_empty[b]);
                }
                // the arithmetic of the other epilogues: round to fp16, then alpha, the residual and ReLU in fp16
#pragma unroll
                for (int i = 0; i < ROWS / 8; ++i)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t* r = (k < 2 ? lo : hi) + 4 * i + 2 * (k & 1);
                        h[i][k] = __hmul2(__floats2half2_rn(__uint_as_float(r[0]), __uint_as_float(r[1])), alpha2);
                    }
            }
            if (!sm100::mbar_wait_warp(&ready[slot], par, cta_abort, p.status_word, SHFLBW_DEVSTAT_TIMEOUT_ACCUM, p.wait_limit)) return;
            const uint32_t tile = slots + slot * (uint32_t)Cfg::SLOT_BYTES;
#pragma unroll
            for (int i = 0; i < ROWS / 8; ++i) {
                uint32_t r[4];
                sm100::ldmatrix_x4_trans(tile + lane_off + i * 1024, r);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h[i][k] = __hadd2(h[i][k], *(__half2*)&r[k]);
                    if (p.relu) h[i][k] = __hmax2(h[i][k], zero2);
                }
                sm100::stmatrix_x4_trans(tile + lane_off + i * 1024, *(uint32_t*)&h[i][0], *(uint32_t*)&h[i][1], *(uint32_t*)&h[i][2], *(uint32_t*)&h[i][3]);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < ROWS / 8; ++i) {
                const uint4 v = *(const uint4*)(smem + (tile - smem_base) + piece_off + i * 1024);
                if (ok) *(uint4*)(dst + (size_t)((uint32_t)(f0 + ch * ROWS + i * 8 + prow) * (uint32_t)p.out_plane)) = v;
            }
            sm100::fence_proxy_async_smem();                   // this warp's accesses before the copies of the refill
            __syncwarp();
            if ((int)(q & 1) != me) {                          // (phases of `done` in order: chunk q's arrival after chunk q - 1's)
                if (q > 0 && !sm100::mbar_wait_warp(done, (q - 1) & 1, cta_abort, p.status_word, SHFLBW_DEVSTAT_TIMEOUT_ACCUM, p.wait_limit)) return;
                if (lane == 0) sm100::mbar_arrive(done);
                if (refills && li_n < nloc) refill(li_n, id, prev);
            }
            ++q;
            prev = slot;
            if (++slot == (uint32_t)NS) { slot = 0; par ^= 1u; }
        }
    }
}

// BIAS: C holds one value per output row (SpMM, added like C with beta = 1) or per filter (SpConv writing
// NHWC in logical order).  Kernels of their own: as a branch of the others it made small products 1-2 %
// slower (256-item launches of 5-9 us, where every instruction is fetched for the first time).
template <int V, int TM, int KS_, int STAGES, int PW, int MODE, int GROUPS_ = 2, int GATHER_ = kGatherCpAsync,
          int EW_ = 8, bool BIAS = false, bool ADDEND = false, int SLOTS = 0>
__global__ void __launch_bounds__(PanelCfg<V, TM, KS_, STAGES, PW, MODE, GROUPS_, GATHER_, EW_, ADDEND, SLOTS>::THREADS, 1)
panel_umma_kernel(const __grid_constant__ PanelParams p) {
    using Cfg = PanelCfg<V, TM, KS_, STAGES, PW, MODE, GROUPS_, GATHER_, EW_, ADDEND, SLOTS>;
    static_assert(SLOTS == 0 || (MODE == kPanelConvChain && !BIAS && !ADDEND), "box epilogue: chained layers with tokens in lanes");
    constexpr int EW = Cfg::EW;                                             // epilogue warps 0..EW-1, MMA warp EW, producers after it
    constexpr bool SWAP = Cfg::SWAP;                                        // rows in TMEM lanes
    constexpr bool NHWC = MODE == kPanelConv || MODE == kPanelConvScatter;
    constexpr bool CONV = NHWC || MODE == kPanelConvChain || MODE == kPanelConvChainRows;  // implicit-GEMM gather
    constexpr bool CHAIN = MODE == kPanelConvChain || MODE == kPanelConvChainRows;
    constexpr bool ROWS_OUT = MODE == kPanelSpmm || MODE == kPanelConvChain; // transposing epilogue: rows out, tokens contiguous
    static_assert(EW == 8 || (ROWS_OUT && Cfg::ACC_COLS >= 128), "16 epilogue warps: transposing epilogue, >= 32 columns per warp");
    constexpr int KS = Cfg::KS, T = Cfg::T;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment: swizzle atoms are addressed by absolute shared-memory address bits.
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* bar_area = smem + Cfg::PIPE_BYTES + Cfg::OUT_BYTES + Cfg::RES_BYTES;
    uint64_t* full_bar = (uint64_t*)bar_area;          // [STAGES] producers -> MMA
    uint64_t* empty_bar = full_bar + STAGES;           // [STAGES] MMA -> producers
    constexpr int NBUF = Cfg::NBUF;
    uint64_t* acc_full = empty_bar + STAGES;           // [NBUF] MMA -> epilogue
    uint64_t* acc_empty = acc_full + NBUF;             // [NBUF] epilogue -> MMA
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + NBUF);
    volatile int* cta_abort = (volatile int*)(tmem_slot + 1);
    uint64_t* drain_bar = acc_empty + NBUF + 1;        // abort path only: MMA thread waits for its last MMAs
    uint64_t* slot_bar = full_bar + STAGES * 2 + 12;   // [SLOT_BARS] box epilogue
    int2* item_tab = (int2*)(bar_area + Cfg::BAR_BYTES);  // [nloc] (first padded row, padded row count)
    int* idx_ring = (int*)(bar_area + Cfg::BAR_BYTES + Cfg::TAB_BYTES);  // [IDX_RING][KS] row ids of upcoming stages

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    // This CTA's work items: blockIdx.x, blockIdx.x + gridDim.x, ...  (host guarantees nloc <= table size)
    const int nloc = (p.num_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    auto item_block = [&](int item) { return p.tile_major ? item - fast_div(item, p.div_blocks) * p.num_blocks : fast_div(item, p.div_tiles); };
    auto item_tile = [&](int item) { return p.tile_major ? fast_div(item, p.div_blocks) : item - fast_div(item, p.div_tiles) * p.tiles_n; };

    if (warp == 0) {                                       // barriers, a lane each
        static_assert(2 * STAGES + 2 * NBUF <= 32, "a barrier per lane");
        // cp.async gather: one arrival per producer WARP of the group (per-thread deferred arrivals,
        // cp.async.mbarrier.arrive.noinc, were measured at ~3 clk of load/store-unit time per thread,
        // i.e. more than the copies themselves).  TMA gather: one arrival per warp of the group too, with the
        // bytes that it fetches, whether it has a row in the stage or not (see the producers).  Stages are emptied by
        // one tcgen05.commit, accumulators by an arrival of each epilogue warp of the set that reads them.
        if (lane < 2 * STAGES + 2 * NBUF)
            sm100::mbar_init(&full_bar[lane], lane < STAGES ? PW / Cfg::GROUPS : lane < 2 * STAGES + NBUF ? 1 : EW / Cfg::ESETS);
        for (int b = lane; b < Cfg::SLOT_BARS; b += 32) sm100::mbar_init(&slot_bar[b], 1);
        if (lane == 0) { sm100::mbar_init(drain_bar, 1); *cta_abort = 0; }
        sm100::mbar_init_fence();
    }
    for (int li = tid; li < nloc; li += blockDim.x) {
        const int blk = item_block((int)blockIdx.x + li * (int)gridDim.x);
        const int b0 = __ldg(p.blk_ptr + blk);
        item_tab[li] = make_int2(b0, __ldg(p.blk_ptr + blk + 1) - b0);
    }
    if (warp == EW) {
        sm100::tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
        sm100::tmem_relinquish();
    }
    const uint32_t smem_base = sm100::smem_u32(smem);
    // The end of the set-up, passed by every warp of the block, in its role: the producers of the TMA gather come with the
    // row ids of their first stages under way.
    // Programmatic dependent launch: everything before (barriers, TMEM, the item table, row ids -- read from
    // the sparse operand, which no kernel writes) may overlap the tail of the previous kernel in
    // the stream; the dense operand, the residual and the output are touched only after the wait below.  The
    // next kernel may start its own prologue as soon as every block of this one got here.
    // (A convolution call that ends with this kernel lets the next one in when its producers have issued, or by
    // cp.async completed, their last copies: early enough for the set-up of an SpMM or a chained layer behind it, about
    // 1 us, and late enough that few blocks of another convolution's relayout, which has no set-up, wait on this kernel's
    // SMs; with those spread evenly (relayout_smem) calls back to back are 1-3 % slower than without any trigger.
    // 24x16x16x160 -> 1856, 3x3, V = 32: 23.9 us and 28.6 with a chained layer; without a trigger 23.7 and 29.8.)
    auto set_up_done = [&]() {
        sm100::tc_fence_before_sync();
        asm volatile("bar.sync 0;" ::: "memory");
        sm100::tc_fence_after_sync();
        if (!NHWC || (MODE == kPanelConv && p.perm != nullptr)) sm100::grid_dependency_launch();
    };
    // The wait itself is executed per role, as late as each role allows: by the producers after
    // their first row ids (sparse operand) are on their way and before their first gather, by the
    // epilogue warps at once (they read C / the residual and write the output); the MMA warp
    // touches no global memory and does not wait.

    const int pidx = Cfg::TMA ? warp - (EW + 1) : warp - (EW + 1) - (warp / 4 - EW / 4);   // producer number of a producer warp (warps after the MMA warp with warp % 4 != 0)
    if (!Cfg::TMA && warp > EW && ((warp & 3) == 0 || pidx >= PW)) {
        set_up_done();                                      // idle: keeps producers off the MMA warp's scheduler partition
    } else if (warp > EW && Cfg::TMA) {
        // ---------------------------------------------------- producers (TMA gather) ----
        // A stage is KS gathered rows x T tokens = (KS/4) row quads x (T/64) column boxes, one
        // tile::gather4 each (4 rows x 128 bytes, landing as half a swizzle atom).  GROUPS groups of GW warps
        // take the stages in turn, a warp's row quads are issued by an elected lane, and the stage's barrier
        // completes by byte count: nobody waits for data.
        // Bound by the issue: an operation takes seven operands in uniform registers, 15 clk of a warp that has
        // the issue slots for itself and 32 in here, where the copy engine would take one every 9.  Hence two
        // warps a stage (11008x4096x512, V = 32, density 0.25: 34.9 us with one, 32.5 with two; 4096^3 at
        // V = 16, 0.1: 77.4 and 72.3; sixteen warps, four to a stage: 33.3 and 74.0), four for SpMM with rows in
        // lanes (4096^3, V = 64: 26.4 us with two, 25.3 with four), and a loop whose control the compiler can see to be uniform.
        // Every warp of a stage arrives on its barrier, with the bytes it fetches.  If only one did, a warp
        // without a row in a short last stage would be waited for by nobody, could fall a whole ring behind,
        // miss the phase that it waits for and wait for good.
        // The CTA's first stage is split between all warps: nothing else is in flight then, and the issue would be
        // most of its time (256^3: 3.1 -> 2.6 us).
        if constexpr (Cfg::TMA) {
        constexpr int BOXES = T / 64, QUADS = KS / 4;       // column boxes per row quad, row quads
        constexpr int GROUPS = Cfg::GROUPS, GW = PW / GROUPS;   // GW warps share a stage
        constexpr int WQ = QUADS / GW;                      // quads of a stage that a warp fetches
        constexpr int IPL = (WQ * 4 + 31) / 32;             // row ids per lane
        const int grp = pidx / GW, pw = pidx % GW;
        int* const my_ids = idx_ring + pidx * KS;           // row ids of this warp's current stage
        if (sm100::elect_one()) sm100::prefetch_tensormap(p.tmap_b);
        // (item, stage of the item) of this warp's next stage; row ids are loaded while the stage before is filled
        int li = 0, kt = 0, row_begin = 0, rows_total = 0;
        auto settle = [&]() {                               // stages beyond an item's end belong to the items after it
            while (li < nloc) {
                const int2 e = item_tab[li];
                row_begin = __shfl_sync(0xffffffffu, e.x, 0); rows_total = __shfl_sync(0xffffffffu, e.y, 0);   // (uniform to the compiler)
                const int num_k = (rows_total + KS - 1) / KS;
                if (kt < num_k) return;
                kt -= num_k;
                ++li;
            }
        };
        auto row_id = [&](int r) {                           // of the item's row r
            int v = li < nloc && r < rows_total ? __ldg(p.blk_idx + row_begin + r) : 0;
            // (SpConv: column ids come decoded as c | r << 16 | s << 24; the map's row is the pixel that the tap starts at)
            if constexpr (CONV) v = ((v & 0xffff) * p.Hp + ((v >> 16) & 0xff)) * p.Wp + ((v >> 24) & 0xff);
            return v;
        };
        int id[IPL];
        auto load_ids = [&]() {
#pragma unroll
            for (int i = 0; i < IPL; ++i) id[i] = row_id(kt * KS + pw * WQ * 4 + i * 32 + lane);
        };
        int xs[BOXES], boxes = 0, nbox = 0, of_item = -1;   // first column of each box; boxes that hold any token
        auto enter_item = [&]() {
            of_item = li;
            const int tok0 = item_tile((int)blockIdx.x + li * (int)gridDim.x) * T;
            boxes = 0;                                       // boxes without a token that is stored are not fetched
#pragma unroll
            for (int b = 0; b < BOXES; ++b) {
                const int tok = tok0 + b * 64;
                xs[b] = tok;
                bool any = tok < p.N;
                if constexpr (CONV) {
                    const int pix = fast_div(tok, p.div_bp), oh = fast_div(pix, p.div_row), ow = pix - oh * p.row_pix;
                    xs[b] = (oh * p.Wp + ow) * p.stride * p.Bp + tok - pix * p.Bp;
                    any = any && ow < p.Wo;
                }
                boxes |= (int)any << b;
            }
            nbox = __popc(boxes);
        };
        // rows in lanes: [K group][T/64 atoms]; tokens in lanes: [128-token half][K group][2 atoms]
        auto dst_off = [](int q, int b) {
            return SWAP ? (uint32_t)((q >> 1) * Cfg::KG_BYTES + b * 1024 + (q & 1) * 512)
                        : (uint32_t)((b >> 1) * Cfg::G_ACC + (q >> 1) * 2048 + (b & 1) * 1024 + (q & 1) * 512);
        };
        auto arm = [&](uint32_t slot, int it, int row0, int rows_valid, int rows_mine) {   // expect this warp's bytes of a stage; the first of its warps copies the value slice
            const uint32_t wbytes = pw == 0 ? (uint32_t)(rows_valid * V * 2) : 0u, bytes = (uint32_t)(rows_mine * nbox * 128) + wbytes;
#ifdef SHFLBW_FAULT_INJECT
            if (p.inject_from >= 0 && it >= p.inject_from) sm100::mbar_expect_tx(&full_bar[slot], bytes);   // the withheld arrival
            else
#endif
            sm100::mbar_arrive_expect_tx(&full_bar[slot], bytes);
            if (pw == 0) sm100::bulk_copy_g2s(smem_base + slot * Cfg::STAGE_BYTES + (uint32_t)Cfg::G_BYTES, p.blk_val + (size_t)row0 * V, wbytes, &full_bar[slot]);
        };
        // The CTA's first stage: this warp's quads of it.  The first item's extent, the ids of these and those of the warp's
        // first whole stage are read beside the block's set-up: a block that starts behind the last ones of the kernel before
        // (grids of every SM) has them 0.5 us earlier (1024x1024x960, V = 32 4.91 -> 4.56 us, 4096^3 at V = 64 25.0 -> 23.4,
        // 28x28x512 -> 128 chained, batch 8, 4.17 -> 3.96; read after the set-up, by its table, and one after the other before).
        constexpr int QW = (QUADS + PW - 1) / PW;
        {
            const int* const ext = p.blk_ptr + item_block((int)blockIdx.x);
            const int e0 = __ldg(ext), e1 = __ldg(ext + 1);
            enter_item();
            row_begin = __shfl_sync(0xffffffffu, e0, 0); rows_total = __shfl_sync(0xffffffffu, e1, 0) - row_begin;
        }
        int first_li = 0, first_row = row_begin, first_valid = min(KS, rows_total), first_id = 0;
        if (lane < QW * 4) first_id = row_id(pidx * QW * 4 + lane);
        kt = 1 + grp;
        const bool in_first = kt * KS < rows_total;
        if (in_first) load_ids();
        set_up_done();
        if (first_valid == 0) {                             // an empty first item: on to one that is not
            kt = 0;
            settle();
            first_li = li; first_row = row_begin;
            if (li < nloc) {
                first_valid = min(KS, rows_total);
                if (lane < QW * 4) first_id = row_id(pidx * QW * 4 + lane);
                enter_item();
            }
            kt += 1 + grp;
        }
        if (!in_first) {
            settle();
            load_ids();
        }
        if (lane < QW * 4) my_ids[lane] = first_id;
        __syncwarp();
        sm100::grid_dependency_wait();                      // the dense operand may be the previous kernel's output
        if (first_li < nloc && sm100::elect_one()) {
            if (grp == 0) arm(0, 0, first_row, first_valid, pw == 0 ? first_valid : 0);
#pragma unroll
            for (int i = 0; i < QW; ++i) {
                const int q = pidx * QW + i;
                const int4 r = *(const int4*)(my_ids + i * 4);
#pragma unroll
                for (int b = 0; b < BOXES; ++b)
                    if (q * 4 < first_valid && (boxes >> b & 1)) sm100::tma_gather4(smem_base + dst_off(q, b), p.tmap_b, xs[b], r.x, r.y, r.z, r.w, &full_bar[0]);
            }
        }
        __syncwarp();
        uint32_t s = 1 + grp, ph = 1;                      // ring slot and the parity that says it is free (in the first lap it is)
        if (s >= (uint32_t)STAGES) { s -= STAGES; ph ^= 1u; }
        int it = 1 + grp;
        while (li < nloc) {
            if (of_item != li) enter_item();
#pragma unroll
            for (int i = 0; i < IPL; ++i) if (WQ * 4 % 32 == 0 || i * 32 + lane < WQ * 4) my_ids[i * 32 + lane] = id[i];
            const int rows_valid = min(KS, rows_total - kt * KS);   // multiple of 16
            const int row0 = row_begin + kt * KS;
            kt += GROUPS;
            settle();
            load_ids();
            if (!sm100::mbar_wait_warp(&empty_bar[s], ph, cta_abort, p.status_word, SHFLBW_DEVSTAT_TIMEOUT_EMPTY, p.wait_limit)) break;
            __syncwarp();                                    // the row ids are in place
            if (sm100::elect_one()) {
                const uint32_t st_base = smem_base + s * Cfg::STAGE_BYTES;
                arm(s, it, row0, rows_valid, min(max(rows_valid - pw * WQ * 4, 0), WQ * 4));
                // All row ids come into registers before the first copy: the copies are ordered with
                // respect to reads of shared memory, which would each add their latency.
                int4 r[WQ];
#pragma unroll
                for (int q = 0; q < WQ; ++q) r[q] = *(const int4*)(my_ids + q * 4);
                auto copy = [&](int q, int b) {
                    sm100::tma_gather4(st_base + pw * (uint32_t)((WQ >> 1) * (SWAP ? Cfg::KG_BYTES : 2048)) + dst_off(q, b), p.tmap_b, xs[b], r[q].x, r[q].y, r[q].z, r[q].w, &full_bar[s]);
                };
                if (rows_valid == KS && nbox == BOXES) {     // a whole stage: straight-line code
#pragma unroll
                    for (int q = 0; q < WQ; ++q)
#pragma unroll
                        for (int b = 0; b < BOXES; ++b) copy(q, b);
                } else {
#pragma unroll
                    for (int q = 0; q < WQ; ++q)
#pragma unroll
                        for (int b = 0; b < BOXES; ++b)
                            if ((pw * WQ + q) * 4 < rows_valid && (boxes >> b & 1)) copy(q, b);
                }
            }
            __syncwarp();                                    // the row ids may be overwritten
            it += GROUPS; s += GROUPS;
            if (s >= (uint32_t)STAGES) { s -= STAGES; ph ^= 1u; }
        }
        if (NHWC && p.trigger_late) sm100::grid_dependency_launch();
        }
    } else if (warp > EW) {
        // --------------------------------------------- producers (cp.async gather) ----
        set_up_done();
        if constexpr (!Cfg::TMA) {
        // The PW producer warps form GROUPS groups that take the CTA's stages in turn (group g
        // fills stages g, g+GROUPS, ...).  While one group sits in its barrier round trip
        // (wait for the free stage, wait for its copies, publish) the other one issues copies,
        // so the load/store unit stays busy; with a single group the round trip (~400 clk)
        // simply added to every stage.
        constexpr int GROUPS = Cfg::GROUPS;
        constexpr int GW = PW / GROUPS;        // warps that share one stage
        constexpr int RPW = KS / GW;           // rows of a stage owned by this warp
        constexpr int CPR = T / 8;             // 16-byte chunks per gathered row
        constexpr int RPI = 32 / CPR;          // rows per warp instruction (TM=2: 1, TM=1: 2)
        constexpr int NQ = RPW / RPI;          // gather copies per lane per stage
        constexpr int XT = NQ < 8 / RPI ? NQ : 8 / RPI;   // period of the swizzle term along q
        static_assert(RPW % 8 == 0 || 8 % RPW == 0, "a producer warp owns whole 8-row swizzle groups or an aligned part of one");
        const int grp = pidx / GW, pw = pidx % GW;
        const int chunk = lane % CPR;          // this lane's chunk of the token tile
        const int sub = RPI == 2 ? (lane >> 4) : 0;
        // Everything that does not change from stage to stage is computed once.  Row q of this
        // lane is r = pw*RPW + q*RPI + sub; its swizzled offset splits into a lane constant, a
        // compile-time term in q and one of XT lane-dependent XOR terms.
        const int rbase = pw * RPW + sub;
        // K group (8 rows) stride and the 64-token swizzle atom inside it.  Tokens as UMMA M: two
        // 128-token halves, each [K group][2 atoms].  Tokens as UMMA N: [K group][T/64 atoms].
        const uint32_t gbase = SWAP ? (uint32_t)((pw * RPW / 8) * Cfg::KG_BYTES + (chunk >> 3) * 1024)
                                    : (uint32_t)((chunk >> 4) * Cfg::G_ACC + (pw * RPW / 8) * 2048 + (((chunk & 15) >> 3)) * 1024);
        uint32_t gx[XT];
#pragma unroll
        for (int j = 0; j < XT; ++j) {
            const int r7 = (pw * RPW + j * RPI + sub) & 7;
            gx[j] = (uint32_t)(r7 * 128 + (((chunk & 7) ^ r7) << 4));
        }
        // A cursor walks the flattened (item, stage) sequence of this CTA using the item table.
        struct Cursor { int li, kt, num_k, row_begin, rows_total; };
        auto enter = [&](Cursor& c) {           // position on the first stage of item c.li (skipping empty items)
            c.kt = 0;
            while (c.li < nloc) {
                const int2 e = item_tab[c.li];
                c.row_begin = e.x; c.rows_total = e.y; c.num_k = (e.y + KS - 1) / KS;
                if (c.num_k > 0) return;
                ++c.li;
            }
            c.num_k = 0; c.row_begin = 0; c.rows_total = 0;
        };
        auto advance = [&](Cursor& c) { if (++c.kt >= c.num_k) { ++c.li; enter(c); } };
        // Row ids are prefetched with 4-byte cp.async into a shared-memory ring (slot = stage %
        // IDX_RING; this warp owns entries [pw*RPW, pw*RPW + RPW) of its group's slots), two of
        // the group's stages ahead: they travel in the first cp.async group of a stage, and the
        // publish step of the group's second stage before the one that reads them is the
        // last wait that is certain to cover that group.
        // (A register prefetch would stall: rotating the registers waits for the load in flight.)
        auto prefetch_idx = [&](const Cursor& c, int stage_no) {
            if (lane < RPW) {
                const int r = c.kt * KS + pw * RPW + lane;
                const bool ok = c.li < nloc && r < c.rows_total;
                sm100::cp_async_4(sm100::smem_u32(idx_ring + (stage_no % Cfg::IDX_RING) * KS + pw * RPW + lane),
                                  ok ? p.blk_idx + c.row_begin + r : p.blk_idx, ok ? 4u : 0u);
            }
        };
        static_assert(RPW <= 32, "one lane per row of the warp's share when prefetching ids");

        Cursor cur{0, 0, 0, 0, 0}, pre{0, 0, 0, 0, 0};
        enter(cur);
        pre = cur;
        for (int d = 0; d < grp; ++d) advance(pre);            // the group's first stage
#pragma unroll 1
        for (int d = 0; d < Cfg::IDX_AHEAD; ++d) {             // ids of its first stages
            prefetch_idx(pre, grp + d * GROUPS);
            for (int g = 0; g < GROUPS; ++g) advance(pre);
        }
        sm100::cp_async_commit();
        sm100::cp_async_wait<0>();
        __syncwarp();
        sm100::grid_dependency_wait();                         // the dense operand may be the previous kernel's output

        int it = 0;        // stage counter across items (all groups count the same sequence)
        int pend = -1;     // this group's stage not yet published
        for (int li = cur.li; li < nloc; ++li) {
            const int2 ent = item_tab[li];
            const int num_k = (ent.y + KS - 1) / KS;
            if (num_k == 0) continue;
            // per-item decode of this lane's tokens
            const int item = (int)blockIdx.x + li * (int)gridDim.x;
            const int tok0 = item_tile(item) * T + chunk * 8;
            const bool chunk_ok = tok0 < p.N;
            const uint32_t nbytes = chunk_ok ? 16u : 0u;
            // SpConv: this lane's 8 tokens are 8 images of one output pixel; the staged input
            // has a zero halo, so tap (r, s) of that pixel is simply base + ((r*Wp + s) * Bp).
            const __half* conv_src0 = p.Xs;
            if constexpr (CONV) {
                if (chunk_ok) {
                    const int pix = fast_div(tok0, p.div_bp), nn = tok0 - pix * p.Bp;
                    const int oh = fast_div(pix, p.div_row), ow = pix - oh * p.row_pix;
                    conv_src0 = p.Xs + ((oh * p.stride * p.Wp + ow * p.stride) * p.Bp + nn);
                }
            }
            const __half* lane_src0 = chunk_ok ? p.B + tok0 : p.B;   // SpMM: column tok0 of row 0
            const uint32_t row_pitch = chunk_ok ? (uint32_t)p.N : 0u;   // out-of-range chunks read B[0] with size 0
            const __half* wsrc = p.blk_val + (size_t)ent.x * V;   // the block's value panel (stage kt at + kt*KS*V)

            for (int kt = 0; kt < num_k; ++kt, ++it) {
                if ((it % GROUPS) != grp) continue;            // the other group's stage
                const int s = it % STAGES, s_idx = it % Cfg::IDX_RING;
                if (it >= STAGES && !sm100::mbar_wait_warp(&empty_bar[s], ((it / STAGES) - 1) & 1, cta_abort, p.status_word,
                                                           SHFLBW_DEVSTAT_TIMEOUT_EMPTY, p.wait_limit))
                    goto producer_done;                        // timed out or aborted: stop issuing
                const int rows_valid = min(KS, ent.y - kt * KS);  // multiple of 16
                const uint32_t st_base = smem_base + s * Cfg::STAGE_BYTES;
                // The group's stage before this one is published half-way through this stage's
                // copies: every stage is committed as two cp.async groups, so "all but the newest
                // group" covers every copy of that stage, issued half an issue phase ago or more.
                auto publish_prev = [&]() {
                    sm100::cp_async_commit();
                    if (pend >= 0) {
                        sm100::cp_async_wait<1>();
                        sm100::fence_proxy_async_smem();   // every lane: its generic-proxy writes -> tensor-core reads
                        __syncwarp();
#ifdef SHFLBW_FAULT_INJECT
                        if (p.inject_from >= 0 && it >= p.inject_from && pidx == 0) return;   // the withheld arrival
#endif
                        if (lane == 0) sm100::mbar_arrive(&full_bar[pend]);
                    }
                };
                // Value panel slice [rows_valid][V]: stored in global memory in the byte order of
                // the shared-memory operand tile, so one bulk copy by the copy engine places it;
                // its bytes are added to what the stage's barrier waits for.
                if (pw == 0 && lane == 0) {
                    const uint32_t wbytes = (uint32_t)(rows_valid * V * 2);
                    sm100::mbar_expect_tx(&full_bar[s], wbytes);
                    sm100::bulk_copy_g2s(st_base + (uint32_t)Cfg::G_BYTES, wsrc + (size_t)kt * KS * V, wbytes, &full_bar[s]);
                }
                prefetch_idx(pre, it + Cfg::IDX_AHEAD * GROUPS);   // joins this iteration's first cp.async group
                for (int g = 0; g < GROUPS; ++g) advance(pre);
                const int* ids = idx_ring + s_idx * KS;  // landed: their group was awaited last iteration

                // All row ids / offsets are fetched into registers BEFORE the first copy: the copy
                // instructions are ordered with respect to shared-memory reads, so a read placed
                // between two copies would serialise its latency into every iteration.
                if constexpr (!CONV) {
                    int idr[NQ];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) idr[q] = (int)min((unsigned)ids[rbase + q * RPI], p.idx_limit);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        if (q == NQ / 2) publish_prev();
                        if (rbase + q * RPI < rows_valid)
                            sm100::cp_async_16(st_base + gbase + (uint32_t)(((q * RPI) >> 3) * Cfg::KG_BYTES) + gx[q % XT],
                                               lane_src0 + (uint64_t)(uint32_t)idr[q] * row_pitch, nbytes);
                    }
                } else {
                    // Column ids arrive decoded (c | r << 16 | s << 24).  Lane j < RPW turns row
                    // pw*RPW + j into an element offset once; the copies fetch it by shuffle.
                    const int idv = ids[pw * RPW + (lane % RPW)];
                    const int delta = (int)min((unsigned)(((idv & 0xffff) * (p.Hp * p.Wp) + ((idv >> 16) & 0xff) * p.Wp + ((idv >> 24) & 0xff)) * p.Bp),
                                               p.idx_limit);
                    int dq[NQ];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) dq[q] = __shfl_sync(0xffffffffu, delta, q * RPI + sub);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        if (q == NQ / 2) publish_prev();
                        if (rbase + q * RPI < rows_valid)
                            sm100::cp_async_16(st_base + gbase + (uint32_t)(((q * RPI) >> 3) * Cfg::KG_BYTES) + gx[q % XT],
                                               conv_src0 + dq[q], nbytes);
                    }
                }
                sm100::cp_async_commit();
                pend = s;
            }
        }
    producer_done:
        // Publish the group's last stages (after a failed wait: just wait for the copies in flight).
        sm100::cp_async_wait<0>();
        sm100::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && pend >= 0) sm100::mbar_arrive(&full_bar[pend]);
        if (NHWC && p.trigger_late) sm100::grid_dependency_launch();
        }
    } else if (warp == EW) {
        // ------------------------------------------------------------ MMA warp ----
        set_up_done();
        const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
        constexpr uint32_t idesc = SWAP ? sm100::make_idesc_f16_mnmajor(V, T) : sm100::make_idesc_f16_mnmajor(128, V);
        // Descriptors are built once; per MMA only the 16-byte-granular start address field
        // (low bits) advances.
        const uint64_t gdesc0 = sm100::make_smem_desc(smem_base, 1024, Cfg::KG_BYTES, sm100::kSwizzle128B);
        const uint64_t wdesc0 =
            V == 16 ? sm100::make_smem_desc(smem_base + Cfg::G_BYTES, 256, 256, sm100::kSwizzle32B)
          : V == 32 ? sm100::make_smem_desc(smem_base + Cfg::G_BYTES, 512, 512, sm100::kSwizzle64B)
          : V == 64 ? sm100::make_smem_desc(smem_base + Cfg::G_BYTES, 1024, 1024, sm100::kSwizzle128B)
                    : sm100::make_smem_desc(smem_base + Cfg::G_BYTES, 1024, 2048, sm100::kSwizzle128B);
        constexpr uint32_t WSTEP = V * 32;  // bytes per K-step (16 rows) of the value tile
        // One elected lane runs the whole role: the ring slot, its parity and the descriptors are then uniform to
        // the compiler, an MMA is a few instructions, and a stage costs 118 clk of this loop plus its MMAs (the
        // warp waiting in lock step and electing per stage: 228; a thread that is not elected, lane == 0: 54 clk per
        // MMA whatever its shape, 1174 clk per stage of the 4096^3 product at V = 64, 1420 at V = 128).
        if (sm100::elect_one()) {
            uint32_t s = 0, ph = 0;     // ring slot of the next stage and the parity of its full barrier
            bool ready = false;         // that barrier was already seen complete
            for (int li = 0; li < nloc; ++li) {
                const int rows_total = item_tab[li].y;
                const int num_k = (rows_total + KS - 1) / KS;
                const int b = li % NBUF;
                if (li >= NBUF && !sm100::mbar_wait_bounded(&acc_empty[b], ((li / NBUF) - 1) & 1, cta_abort, p.status_word,
                                                            SHFLBW_DEVSTAT_TIMEOUT_ACCUM, p.wait_limit))
                    break;                                   // timed out or aborted: issue nothing more
                const uint32_t acc_base = tmem_base + b * Cfg::ACC_COLS;
                for (int kt = 0; kt < num_k; ++kt) {
                    if (!ready && !sm100::mbar_wait_bounded(&full_bar[s], ph, cta_abort, p.status_word, SHFLBW_DEVSTAT_TIMEOUT_FULL, p.wait_limit))
                        goto mma_done;                       // timed out or aborted: issue nothing more
                    // cp.async (generic proxy) data -> tensor-core (async proxy) reads; the copy engine's
                    // writes of the TMA gather are in the async proxy already
                    if (!Cfg::TMA) sm100::fence_proxy_async_smem();
                    sm100::tc_fence_after_sync();
                    const uint32_t sn = s + 1 == (uint32_t)STAGES ? 0 : s + 1;
                    ready = sm100::mbar_test(&full_bar[sn], sn ? ph : ph ^ 1u);   // the round trip hides behind the MMAs
                    const int nk = min(KS, rows_total - kt * KS) / 16;
                    const uint64_t gd = gdesc0 + (uint64_t)((s * (uint32_t)Cfg::STAGE_BYTES) >> 4);
                    const uint64_t wd = wdesc0 + (uint64_t)((s * (uint32_t)Cfg::STAGE_BYTES) >> 4);
#pragma unroll
                    for (int j = 0; j < KS / 16; ++j) {
                        if (j < nk) {
                            const uint64_t gdj = gd + (uint64_t)(j * ((2 * Cfg::KG_BYTES) >> 4)), wdj = wd + (uint64_t)(j * (WSTEP >> 4));
                            const uint32_t accum = j > 0 || kt > 0;
                            if constexpr (SWAP) {
                                // D[row][token] += W^T . G
                                if constexpr (Cfg::WS) sm100::umma_ws_f16_ss(acc_base, wdj, gdj, idesc, accum);
                                else sm100::umma_f16_ss(acc_base, wdj, gdj, idesc, accum);
                            } else {
#pragma unroll
                                for (int a = 0; a < TM; ++a)
                                    sm100::umma_f16_ss(acc_base + a * V, gdj + (uint64_t)((a * Cfg::G_ACC) >> 4), wdj, idesc, accum);
                            }
                        }
                    }
                    sm100::umma_commit(&empty_bar[s]);       // stage may be refilled once these MMAs retire
                    if (kt + 1 == num_k) sm100::umma_commit(&acc_full[b]);   // accumulator complete
                    s = sn;
                    if (sn == 0) ph ^= 1u;
                }
                if (num_k == 0) sm100::mbar_arrive(&acc_full[b]);   // nothing to wait for
            }
        mma_done:
            if (*cta_abort) {
                // Aborted: the MMAs issued so far must retire before TMEM is freed and the block's
                // shared memory goes away.  One more commit, awaited with its own (short) limit.
                sm100::umma_commit(drain_bar);
                sm100::mbar_wait_bounded(drain_bar, 0, cta_abort, p.status_word, 0, 4000000LL, /*heed_abort=*/false);
            }
        }
        __syncwarp();
    } else {
        // -------------------------------------------------------------- epilogue ----
        // Warp w reads TMEM lane quadrant w % 4 (tokens) and half w / 4 % 2 of the accumulator
        // columns (the block's output rows / filters).  Sixteen warps are two sets of eight that take
        // the items in turn: against all sixteen on one item (a quarter of the columns each), 108 ->
        // 93 us on 56x56x64 -> 256 at batch 256, since an item's chain of waits is most of its time.
        set_up_done();
        const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
        sm100::grid_dependency_wait();
        if constexpr (SLOTS > 0) {
            box_epilogue<Cfg, V>(p, smem, smem_base, tmem_base, item_tab, nloc, acc_full, acc_empty, slot_bar, cta_abort, warp, lane, item_block, item_tile);
        } else {
        const int quad = warp & 3, half_id = (warp >> 2) & 1;
        // (a single 16- or 32-column accumulator is not split; two 16-column accumulators go to the two halves)
        constexpr int HALVES = (Cfg::ACC_COLS >= 64 || (V == 16 && TM == 2)) ? 2 : 1;
        constexpr int COLS = Cfg::ACC_COLS / HALVES;          // fp32 columns handled by this warp
        constexpr int CW = COLS < 32 ? COLS : 32;             // columns per pass through the 2 KB tile
        const bool reads = half_id < HALVES;
        const __half alpha1 = __float2half_rn(p.alpha), beta1 = __float2half_rn(p.beta);
        const __half2 alpha2 = __half2half2(alpha1);
        bool res_primed = false;               // addend copies (RES_BYTES) run an item ahead
        for (int li = Cfg::ESETS > 1 ? warp >> 3 : 0; li < nloc; li += Cfg::ESETS) {
            const int item = (int)blockIdx.x + li * (int)gridDim.x;
            const int blk = item_block(item);
            const int n0 = item_tile(item) * T;
            const bool has_k = item_tab[li].y > 0;
            const int b = li % NBUF;
            // Wait for the item's accumulator (the whole warp).  false: the wait
            // timed out or the block is aborting -- store nothing more.
            auto wait_accumulator = [&]() -> bool {
                if (!sm100::mbar_wait_warp(&acc_full[b], (li / NBUF) & 1, cta_abort, p.status_word,
                                           SHFLBW_DEVSTAT_TIMEOUT_ACCUM, p.wait_limit))
                    return false;
                sm100::tc_fence_after_sync();
                return true;
            };
            // Rows in lanes: the bias of this lane's row is one value for the whole item, requested before the
            // wait, which hides its two dependent loads; the stores stay the wide ones.  (Looked up for every
            // 8 tokens, after the accumulator read: a 4096 x 4096 layer, V = 64, density 0.1, of 4096 tokens
            // took 68.0 us with a bias and 45.7 without; 45.7 now.)
            __half2 bias2 = __float2half2_rn(0.f);
            if constexpr (SWAP && BIAS) {
                const int m = (Cfg::WS ? quad & 1 : quad) * 32 + lane;
                bias2 = __half2half2(__ldg(p.C + (p.perm ? __ldg(p.perm + blk * V + m) : blk * V + m)));
            }
            if constexpr (SWAP || !ROWS_OUT) {
                if (!wait_accumulator()) break;
            }
            if constexpr (SWAP) {
                // Rows in lanes: lane l of quadrant `quad` holds output row m of the block (V = 128:
                // m = 32*quad + l; V = 64: m = 32*(quad % 2) + l, the upper two quadrants the second half of the
                // tokens), and the quadrant's two warps share its token columns, 32 at a time: a lane's 32
                // tokens are 64 contiguous bytes of its output row.  They are packed to fp16 and
                // stored straight from registers -- as two 32-byte stores (whole L2 sectors) when
                // the output rows are 32-byte aligned, else as four 16-byte stores.  No shared
                // memory is involved: the tensor core's operand reads and the gather's writes already
                // use most of its bandwidth.
                constexpr int HC = (int)Cfg::ACC_COLS / 2;               // token columns of this warp
                const uint32_t acc0 = tmem_base + ((uint32_t)(quad * 32) << 16) + b * Cfg::ACC_COLS + half_id * HC;
                const int t0 = n0 + (Cfg::WS ? (quad >> 1) * (T / 2) : 0) + half_id * HC;   // its first token
                const int m = (Cfg::WS ? quad & 1 : quad) * 32 + lane;
                size_t roff;                                             // element offset of this lane's output row
                size_t rres = 0;                                         // chained: offset of its residual row
                const bool use_res = CHAIN && p.res != nullptr;
                if constexpr (CHAIN) {
                    // plane of this filter: stored order between chained layers, logical order when the
                    // planes are about to be transposed to NHWC
                    const int plane = (p.out_logical && p.perm) ? __ldg(p.perm + blk * V + m) : blk * V + m;
                    roff = (size_t)plane * (size_t)p.out_plane;
                    if (use_res) rres = (size_t)(p.res_map ? __ldg(p.res_map + blk * V + m) : blk * V + m) * (size_t)p.out_plane;
                } else {
                    const int drow = (p.perm) ? __ldg(p.perm + blk * V + m) : blk * V + m;
                    roff = (size_t)drow * (size_t)p.N;
                }
                __half* const obase = CHAIN ? p.out : p.D;
                const __half2 zero2 = __float2half2_rn(0.f);
                const bool use_c = !CHAIN && !BIAS && p.beta != 0.0f && p.C != nullptr;
#pragma unroll 1
                for (int cc = 0; cc < HC; cc += 32) {
                    const int tok0 = t0 + cc;                            // this lane's 32 tokens start here
                    // Where the four 8-token groups go, and (chained layers) the residual that gets added
                    // to them: requested before the accumulator read, so that the global-memory latency
                    // hides behind it.
                    size_t goffs[4];
                    bool valid[4] = {};
                    uint4 addend[4];
                    {
                        if constexpr (CHAIN) {
                            // 8 consecutive tokens are 8 images of one output pixel; the pixel's place in the
                            // consumer's halo-padded plane is found once and stepped from group to group
                            int pix = fast_div(tok0, p.div_bp), nn = tok0 - pix * p.Bp;
                            int oh = fast_div(pix, p.div_row), ow = pix - oh * p.row_pix;
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                goffs[c] = (size_t)(((oh + p.oph) * p.OWp + ow + p.opw) * p.Bp + nn);
                                valid[c] = tok0 + c * 8 < p.N && ow < p.Wo;
                                nn += 8;
                                if (nn >= p.Bp) { nn = 0; if (++ow >= p.row_pix) { ow = 0; ++oh; } }
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c) goffs[c] = (size_t)(tok0 + c * 8);   // (folds into the addresses)
                        }
                        if constexpr (CHAIN) {
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                addend[c] = make_uint4(0u, 0u, 0u, 0u);
                                if (use_res && valid[c]) addend[c] = *(const uint4*)(p.res + rres + goffs[c]);
                            }
                        }
                    }
                    uint32_t r[32];
                    if (has_k) {
                        sm100::tmem_ld_32x32b_x32(acc0 + cc, r);
                        sm100::tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int e = 0; e < 32; ++e) r[e] = 0u;
                    }
                    if (cc + 32 >= HC) {  // last TMEM read of this item by this warp: release the buffer
                        sm100::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) sm100::mbar_arrive(&acc_empty[b]);
                    }
                    {
                    uint4 v[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        __half2* h = (__half2*)&v[c];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            // same arithmetic as the reference: round to fp16, then alpha in fp16
                            h[e] = __floats2half2_rn(__uint_as_float(r[c * 8 + 2 * e]), __uint_as_float(r[c * 8 + 2 * e + 1]));
                            if constexpr (BIAS) h[e] = __hfma2(h[e], alpha2, bias2);
                            else if (!use_c) h[e] = __hmul2(h[e], alpha2);
                        }
                    }
                    if constexpr (!CHAIN) {
                        __half* dst = obase + roff + tok0;
                        if (p.wide_stores && !use_c) {                   // N % 16 == 0: 16 tokens are valid as a whole
                            if (tok0 < p.N) sm100::st_global_32B(dst, v[0], v[1]);
                            if (tok0 + 16 < p.N) sm100::st_global_32B(dst + 16, v[2], v[3]);
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                if (tok0 + c * 8 < p.N) {                // N % 8 == 0: 8 tokens are valid as a whole
                                    if (use_c) {                         // (the rare beta != 0 case pays the load's latency here)
                                        const uint4 cv = *(const uint4*)(p.C + roff + tok0 + c * 8);
                                        __half* h = (__half*)&v[c];
                                        const __half* ch = (const __half*)&cv;
#pragma unroll
                                        for (int e = 0; e < 8; ++e) h[e] = __hfma(h[e], alpha1, __hmul(ch[e], beta1));
                                    }
                                    *(uint4*)(dst + c * 8) = v[c];
                                }
                            }
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            if (valid[c]) {
                                __half2* h = (__half2*)&v[c];
                                if (use_res) {                           // out = relu(alpha * conv + residual), fp16
                                    const __half2* rh = (const __half2*)&addend[c];
#pragma unroll
                                    for (int e = 0; e < 4; ++e) h[e] = __hadd2(h[e], rh[e]);
                                }
                                if (p.relu) {
#pragma unroll
                                    for (int e = 0; e < 4; ++e) h[e] = __hmax2(h[e], zero2);
                                }
                                *(uint4*)(obase + roff + goffs[c]) = v[c];
                            }
                        }
                    }
                    }
                    __syncwarp();                                        // the next TMEM load is warp-wide
                }
                continue;
            }
            // columns [col0, col0 + COLS) of the accumulator set: accumulator a = col / V, row m = col % V
            const int col0 = half_id * COLS;
            const uint32_t acc_base = tmem_base + ((uint32_t)(quad * 32) << 16) + b * Cfg::ACC_COLS + col0;
            // per-item, per-thread constants
            const int a0 = col0 / V;                       // this warp's columns lie in one accumulator
            const int tok = reads ? n0 + a0 * 128 + quad * 32 + lane : p.N;   // idle warps store nothing
            const int mbase = col0 % V;                    // first block row / filter of this warp
            bool ok = tok < p.N;
            uint32_t row_off[4], position = 0;             // SpConv: output offsets of positions i*8 + lane/4, of this lane's
            int positions = 0, nth = 0;
            if constexpr (NHWC) {
                const int pix = fast_div(tok, p.div_bp), img = tok - pix * p.Bp;
                const int oh = fast_div(pix, p.div_row), ow = pix - oh * p.row_pix;
                ok = ok && img < p.Bn && ow < p.Wo;
                // this position's F-vector at the block's filters (element offset; host checks it fits 32 bits)
                const uint32_t mine = ok ? (uint32_t)((img * p.Ho + oh) * p.Wo + ow) * (uint32_t)p.F + (uint32_t)(blk * V + mbase)
                                         : 0xffffffffu;
#pragma unroll
                for (int i = 0; i < 4; ++i) row_off[i] = __shfl_sync(0xffffffffu, mine, i * 8 + (lane >> 2));
                if constexpr (MODE == kPanelConvScatter) {
                    position = mine - (uint32_t)(blk * V + mbase);
                    const unsigned live = __ballot_sync(0xffffffffu, ok);    // not those of images beyond the batch, pixels beyond a row
                    positions = __popc(live);
                    nth = (int)__fns(live, 0, lane + 1);                     // the lane of the l-th of them (-1: fewer)
                }
            }
            const bool use_c = MODE == kPanelSpmm && (EW == 8 || BIAS || Cfg::RES_BYTES > 0) && p.beta != 0.0f && p.C != nullptr;
            if constexpr (ROWS_OUT) {
            // TMEM lanes are tokens, accumulator columns the block's output rows.  For a fixed row a
            // warp's 32 tokens are only 64 contiguous bytes of D, so each chunk of 32 rows is transposed
            // through a tile in shared memory and comes back as 16-byte pieces: four lanes store one
            // row's 64 bytes, eight rows per store instruction.  The inverse row permutation is the row
            // index of those stores.
            //   64 and 128 rows (TILES): the chunk leaves TMEM as 8 x 8 tiles, which stmatrix writes,
            // transposed, as [row][32 tokens] (the 16-byte chunk c of row r at c ^ (r / 2 % 4): no bank
            // conflicts either way).
            //   16 and 32 rows: 16 row PAIRS x 32 tokens of half2, thread = token (one packed conversion,
            // one multiply and one 4-byte conflict-free write per pair); a lane reads 8 tokens of a pair
            // (two 16-byte reads, the 16-byte units of odd pairs swapped so that a quarter warp covers all
            // banks) and splits them into the pair's two rows with byte permutes.
            // Pairs and tiles, us: SpMM 4096x512x8192, V = 64, 51 columns a block 20.4 and 18.9, 4096x1024x4096 12.6 and
            // 11.7; chained 56x56x64 -> 64, 3x3, batch 256 38.2 and 36.8; V = 128, 28x28x128 -> 256, batch 64, with
            // residual 14.5 and 13.7, batch 8 5.1 and 4.35 (its TMA kernel does not spill any more); V = 32,
            // 11008x4096x512 32.7 and 33.2, 256x256x256 2.78 and 2.93; V = 16, 3072x768x1000 14.5 and 14.9.
            constexpr bool TILES = V >= 64;
            uint8_t* const my_tile = smem + Cfg::PIPE_BYTES + warp * 2048;
            const int tg = lane & 3;                                    // 8-token group stored by this lane
            // stmatrix: lane 8 k + j names tokens 8 k.. of row 8 i + j
            const uint32_t st_off = sm100::smem_u32(my_tile) + (uint32_t)((lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4));
            const uint8_t* const piece = my_tile + (lane >> 2) * 64 + ((tg ^ ((lane >> 3) & 3)) << 4);
            // Row of a chunk that this lane's j-th piece is of (pairs: j = 2i + h is half h of pair 8i + lane/4).
            auto slot_row = [&](int j) { return TILES ? 8 * j + (lane >> 2) : 16 * (j >> 1) + 2 * (lane >> 2) + (j & 1); };
            constexpr int NSLOT = CW / 8;                               // rows stored per lane and chunk
            // This lane's 8-token group of an item whose tile starts at token n0_: is it inside N
            // (N % 8 == 0: a group is valid as a whole), and its element offset inside an output
            // row.  SpMM: the token index.  Chained SpConv: 8 images of one output pixel inside the
            // next layer's halo-padded plane (images beyond the batch are computed from zero inputs
            // and are written as zeros).
            auto group_offset = [&](int n0_, bool& ok_) -> uint32_t {
                const int tok_g = reads ? n0_ + a0 * 128 + quad * 32 + tg * 8 : p.N;
                ok_ = tok_g < p.N;
                uint32_t goff_ = (uint32_t)tok_g;
                if constexpr (MODE == kPanelConvChain) {
                    if (ok_) {
                        const int pix = fast_div(tok_g, p.div_bp), nn = tok_g - pix * p.Bp;
                        const int oh = fast_div(pix, p.div_row), ow = pix - oh * p.row_pix;
                        ok_ = ow < p.Wo;
                        goff_ = (uint32_t)(((oh + p.oph) * p.OWp + ow + p.opw) * p.Bp + nn);
                    }
                }
                return goff_;
            };
            bool ok_g;
            const uint32_t goff = group_offset(n0, ok_g);
            __half* const obase = MODE == kPanelSpmm ? p.D : p.out;
            const __half2 zero2 = __float2half2_rn(0.f);
            // What gets added to the product (beta * C, or the residual of a chained layer) does not
            // depend on the accumulator and is requested early, so that its global-memory latency is off
            // the critical path (these layers are often all epilogue).
            //   Sixteen epilogue warps: an item ahead, by cp.async into the lane's own slots in shared
            // memory.  Ordinary loads would need an L1 line per piece until it arrives, and beside a
            // block's shared memory the L1 holds about 28 KB, less than one item's 32 KB: with them more
            // requests in flight made these layers slower (56x56x64 -> 256 with residual, batch 256:
            // 214 us with loads before the accumulator wait, 230 with two items' loads in flight, 187 with
            // the copies; the same product without a residual takes 93.  All in the executed stack; back to back
            // with the L2 warm 168 and 91).
            //   Eight: into registers, the first two chunks before the accumulator wait, each later
            // chunk's two chunks ahead.
            constexpr int NCH = COLS / CW;
            constexpr bool RES_AHEAD = Cfg::RES_BYTES > 0;
            constexpr bool IN_REGS = EW == 8;     // (sixteen warps without ADDEND add nothing but a bias)
            const bool ahead = RES_AHEAD && ((use_c && !BIAS) || (MODE == kPanelConvChain && p.res != nullptr));
            const bool add_res = (IN_REGS || RES_AHEAD) && MODE == kPanelConvChain && p.res != nullptr;
            const bool need_add = ok_g && (use_c || add_res);
            auto addend_at = [&](int blk_, uint32_t goff_, int cc, int i) -> const __half* {
                const int m = mbase + cc + slot_row(i);
                if (use_c) {
                    const int row = (p.perm) ? __ldg(p.perm + blk_ * V + m) : blk_ * V + m;
                    if constexpr (BIAS) return p.C + row;
                    return p.C + (size_t)((uint32_t)row * (uint32_t)p.N) + (size_t)goff_;
                }
                const uint32_t rr = (uint32_t)(p.res_map ? __ldg(p.res_map + blk_ * V + m) : blk_ * V + m) * (uint32_t)p.out_plane;
                return p.res + (size_t)rr + (size_t)goff_;
            };
            uint4 addend[NCH > 1 && IN_REGS ? 2 : 1][4];
            auto fetch_addend = [&](int blk_, uint32_t goff_, int cc, uint4 (&dst)[4]) {
#pragma unroll
                for (int i = 0; i < NSLOT; ++i) {
                    const __half* src = addend_at(blk_, goff_, cc, i);
                    if constexpr (MODE == kPanelSpmm && BIAS) dst[i] = broadcast8(src);
                    else dst[i] = *(const uint4*)src;
                }
            };
            uint8_t* const my_res = smem + Cfg::PIPE_BYTES + Cfg::OUT_BYTES + warp * 4096 + lane * 16;   // slot (chunk, i): + (chunk*4 + i) * 512
            static_assert(!RES_AHEAD || NCH * NSLOT * 512 <= 4096, "addend slots");
            auto copy_addend = [&](int blk_, uint32_t goff_, bool ok_, int ch_) {   // one cp.async group per chunk, empty or not
                if (ok_) {
#pragma unroll
                    for (int i = 0; i < NSLOT; ++i)
                        sm100::cp_async_16(sm100::smem_u32(my_res + (ch_ * 4 + i) * 512), addend_at(blk_, goff_, ch_ * CW, i), 16u);
                }
                sm100::cp_async_commit();
            };
            int blk_next = 0;                     // this warp's next item: block, group offset, anything to copy
            uint32_t goff_next = 0;
            bool ok_next = false;
            if constexpr (RES_AHEAD) {
                if (ahead) {
                    if (!res_primed) {            // the warp's first item: nothing was copied ahead
#pragma unroll
                        for (int ch = 0; ch < NCH; ++ch) copy_addend(blk, goff, ok_g, ch);
                        res_primed = true;
                    }
                    if (li + Cfg::ESETS < nloc) {
                        const int item_next = (int)blockIdx.x + (li + Cfg::ESETS) * (int)gridDim.x;
                        blk_next = item_block(item_next);
                        goff_next = group_offset(item_tile(item_next) * T, ok_next);
                    }
                }
            } else if (IN_REGS && need_add) {
                fetch_addend(blk, goff, 0, addend[0]);
                if constexpr (NCH > 1 && IN_REGS) fetch_addend(blk, goff, CW, addend[1]);
            }
            if (!wait_accumulator()) break;
#pragma unroll
            for (int ch = 0; ch < NCH; ++ch) {
                const int cc = ch * CW;
                uint32_t roff[4];                                        // D offsets of this lane's rows
#pragma unroll
                for (int i = 0; i < NSLOT; ++i) {
                    const int m = mbase + cc + slot_row(i);
                    if constexpr (MODE == kPanelSpmm) {
                        const int row = (p.perm) ? __ldg(p.perm + blk * V + m) : blk * V + m;
                        roff[i] = (uint32_t)row * (uint32_t)p.N;
                    } else {
                        const int plane = (p.out_logical && p.perm) ? __ldg(p.perm + blk * V + m) : blk * V + m;
                        roff[i] = (uint32_t)plane * (uint32_t)p.out_plane;           // stored (chained) or logical order
                    }
                }
                if constexpr (TILES) {
                    uint32_t lo[CW / 2], hi[CW / 2];      // the chunk's columns of lanes 0-15 and 16-31 of the quadrant
                    if (has_k && reads) {
                        sm100::tmem_ld_16x256b(acc_base + cc, lo);
                        sm100::tmem_ld_16x256b(acc_base + (16u << 16) + cc, hi);
                        sm100::tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int e = 0; e < CW / 2; ++e) lo[e] = hi[e] = 0u;
                    }
                    if (cc + CW >= COLS) {  // last TMEM read of this item by this warp: release the buffer
                        sm100::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) sm100::mbar_arrive(&acc_empty[b]);
                    }
                    // Same epilogue arithmetic as the reference: round to fp16, then alpha (and
                    // beta * C, applied after the transpose) in fp16.
#pragma unroll
                    for (int i = 0; i < NSLOT; ++i) {     // rows 8 i..: four tiles of eight tokens
                        __half2 h[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t* r = (k < 2 ? lo : hi) + 4 * i + 2 * (k & 1);
                            h[k] = __floats2half2_rn(__uint_as_float(r[0]), __uint_as_float(r[1]));
                            if (!use_c) h[k] = __hmul2(h[k], alpha2);
                        }
                        sm100::stmatrix_x4_trans(st_off + i * 512, *(uint32_t*)&h[0], *(uint32_t*)&h[1], *(uint32_t*)&h[2], *(uint32_t*)&h[3]);
                    }
                } else {
                    uint32_t r[CW];                       // the chunk's accumulator columns of this token
                    if (has_k && reads) {
                        if constexpr (CW == 32) sm100::tmem_ld_32x32b_x32(acc_base + cc, r);
                        else sm100::tmem_ld_32x32b_x16(acc_base + cc, r);
                        sm100::tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int e = 0; e < CW; ++e) r[e] = 0u;
                    }
                    if (cc + CW >= COLS) {
                        sm100::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) sm100::mbar_arrive(&acc_empty[b]);
                    }
#pragma unroll
                    for (int q = 0; q < CW / 2; ++q) {
                        __half2 h = __floats2half2_rn(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
                        if (!use_c) h = __hmul2(h, alpha2);
                        ((uint32_t*)my_tile)[q * 32 + (lane ^ ((q & 1) << 2))] = *(uint32_t*)&h;
                    }
                }
                __syncwarp();
                if constexpr (RES_AHEAD) {
                    if (ahead) {
                        sm100::cp_async_wait<NCH - 1>();     // this chunk's copies (each lane reads only its own)
#pragma unroll
                        for (int i = 0; i < NSLOT; ++i) addend[0][i] = *(const uint4*)(my_res + (ch * 4 + i) * 512);
                    }
                }
                if constexpr (BIAS && !IN_REGS) { if (need_add) fetch_addend(blk, goff, cc, addend[0]); }
                {
                    uint4 w0, w1;                            // pairs: 8 tokens of a row pair
#pragma unroll
                    for (int i = 0; i < NSLOT; ++i) {
                        uint4 v;
                        if constexpr (TILES) {
                            v = *(const uint4*)(piece + i * 512);
                        } else {
                            if (i % 2 == 0) {
                                const int q = 4 * i + (lane >> 2);
                                const uint32_t* src = (const uint32_t*)my_tile + q * 32;
                                w0 = *(const uint4*)(src + (((2 * tg) ^ (q & 1)) << 2));
                                w1 = *(const uint4*)(src + (((2 * tg + 1) ^ (q & 1)) << 2));
                            }
                            const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;   // the pair's second / first row
                            v.x = __byte_perm(w0.x, w0.y, sel); v.y = __byte_perm(w0.z, w0.w, sel);
                            v.z = __byte_perm(w1.x, w1.y, sel); v.w = __byte_perm(w1.z, w1.w, sel);
                        }
                        if (ok_g) {
                            const size_t off = (size_t)roff[i] + (size_t)goff;
                            if (use_c) {
                                __half* h = (__half*)&v;
                                const __half* cadd = (const __half*)&addend[NCH > 1 && IN_REGS ? (ch & 1) : 0][i];
#pragma unroll
                                for (int e = 0; e < 8; ++e) h[e] = __hfma(h[e], alpha1, __hmul(cadd[e], beta1));
                            }
                            if constexpr (MODE == kPanelConvChain) {   // out = relu(alpha * conv + residual), fp16
                                __half2* h = (__half2*)&v;
                                if (add_res) {
                                    const __half2* rh = (const __half2*)&addend[NCH > 1 && IN_REGS ? (ch & 1) : 0][i];
#pragma unroll
                                    for (int e = 0; e < 4; ++e) h[e] = __hadd2(h[e], rh[e]);
                                }
                                if (p.relu) {
#pragma unroll
                                    for (int e = 0; e < 4; ++e) h[e] = __hmax2(h[e], zero2);
                                }
                            }
                            *(uint4*)(obase + off) = v;
                        }
                    }
                }
                if constexpr (RES_AHEAD) { if (ahead) copy_addend(blk_next, goff_next, ok_next, ch); }
                else if constexpr (NCH > 2 && IN_REGS) { if (need_add && ch + 2 < NCH) fetch_addend(blk, goff, cc + 2 * CW, addend[ch & 1]); }
                __syncwarp();
            }
            } else {
            // SpConv: thread = output position, accumulator columns = consecutive filters of the
            // block, contiguous in the position's F-vector (stored filter order).  Straight from
            // registers a warp store would touch 32 lines (one per position); instead each
            // 32-filter chunk goes through a swizzled 2 KB tile so that four lanes write one
            // position's 64 contiguous bytes.
            uint8_t* my_tile = smem + Cfg::PIPE_BYTES + warp * 2048;
#pragma unroll 1
            for (int cc = 0; cc < COLS; cc += CW) {
#pragma unroll
                for (int j = 0; j < CW / 8; ++j) {
                    const int c0 = cc + j * 8;
                    uint32_t r[8];
                    if (has_k && reads) {
                        sm100::tmem_ld_32x32b_x8(acc_base + c0, r);
                        sm100::tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) r[e] = 0u;
                    }
                    if (c0 + 8 >= COLS) {  // last TMEM read of this item by this warp: release the buffer
                        sm100::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) sm100::mbar_arrive(&acc_empty[b]);
                    }
                    uint4 v;
                    __half2* h = (__half2*)&v;
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        h[e] = __hmul2(__floats2half2_rn(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), alpha2);
                    *(uint4*)(my_tile + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = v;
                }
                __syncwarp();
                if constexpr (MODE == kPanelConvScatter) {
                    // Filters in logical order without a further pass: lane = filter of the chunk, one position's (CW = 16: two
                    // positions') values to wherever they belong in its F-vector.  Bound by partial sectors at the L2, about
                    // 80 a clock (5x14x14 positions of 512 filters: 2.3 us for 320,000).
                    constexpr int PER = 32 / CW;                         // positions of a store
                    const int f = __ldg(p.perm + blk * V + mbase + cc + lane % CW);
                    const uint32_t e = (uint32_t)(lane % CW);
                    const __half add = p.C ? p.C[f] : __float2half(-0.f);   // (v + -0 is v, also for v = -0)
                    for (int i = 0; i < positions; i += 8 * PER) {       // eight stores' values first (one by one: 120 clocks each)
                        int at[8];
                        uint32_t to[8];
                        __half v[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) at[j] = __shfl_sync(0xffffffffu, nth, i + j * PER + lane / CW);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int row = at[j] & 31;
                            to[j] = __shfl_sync(0xffffffffu, position, row);
                            v[j] = *(const __half*)(my_tile + row * 64 + (((e >> 3) ^ ((row >> 1) & 3)) << 4) + (e & 7) * 2);
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (at[j] >= 0) p.out[(size_t)to[j] + f] = __hadd(v[j], add);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = i * 8 + (lane >> 2), c = lane & 3;
                        uint4 v = *(const uint4*)(my_tile + row * 64 + ((c ^ ((row >> 1) & 3)) << 4));
                        if (BIAS && c < CW / 8) {                        // (stored order is logical order here)
                            const uint4 bv = __ldg((const uint4*)(p.C + blk * V + mbase + cc + c * 8));
                            __half2* h = (__half2*)&v;
                            const __half2* bh = (const __half2*)&bv;
#pragma unroll
                            for (int e = 0; e < 4; ++e) h[e] = __hadd2(h[e], bh[e]);
                        }
                        if (row_off[i] != 0xffffffffu && c < CW / 8) *(uint4*)(p.out + (size_t)row_off[i] + cc + c * 8) = v;
                    }
                }
                __syncwarp();
            }
            }
        }
        if constexpr (Cfg::RES_BYTES > 0) sm100::cp_async_wait<0>();   // nothing of this warp is in flight when the block ends
        }
    }

    if (*cta_abort) {
        // A wait gave up somewhere in this block.  Every role has stopped issuing work, and cp.async copies were
        // awaited above; what is still in flight -- bulk copies of value slices and tile gathers, at most a ring
        // of stages, whose barriers nobody waits for any more -- gets a bounded ~100 us after each thread's last
        // instruction to land before the shared memory is released.
        const long long t0 = clock64();
        while (clock64() - t0 < 200000LL) __nanosleep(1000);
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    if (warp == EW) {
        sm100::tc_fence_after_sync();
        sm100::tmem_dealloc(__shfl_sync(0xffffffffu, *tmem_slot, 0), Cfg::TMEM_COLS);
    }
}


}  // namespace shflbw
