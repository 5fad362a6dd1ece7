// CUDA side of the C ABI: device upload of the Shfl-BW images, op init / exec for SpMM and
// SpConv, and the end-to-end host-buffer calls.  Host code here only validates, fills POD
// states and launches; all arithmetic happens in the kernels of panel_umma.cuh /
// aux_kernels.cuh.  There is no CPU fallback: without a CUDA device every op entry point
// returns SHFLBW_ERR_CUDA.
//
// Reference host code this replaces (paths relative to the reference project):
//   block_sparse/spmm/blockwise_format.h:200-266   transform_and_sync_device
//   block_sparse/spmm/blockwise_op.h:73-132, 169-209   initialize / operator() / InitFn / ExecFn
//   block_sparse/spconv/blockwise_op.h:70-131, 148-187

#include <cuda.h>

#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <utility>

#include "aux_kernels.cuh"
#include "linear_direct.cuh"
#include "panel_umma.cuh"
#include "shflbw_internal.hpp"

namespace {

thread_local char g_cuda_err[256] = "";

// Bound of the kernels' barrier waits in SM clocks, and (fault-injection builds) the stage from
// which one producer warp withholds its arrivals.  Process-wide; read when a launch is issued.
long long g_wait_limit = shflbw::kWaitLimitCycles;
int g_inject_from = -1;
#ifdef SHFLBW_FAULT_INJECT
int g_set_ups_left = -1;             // test builds: this many more shared-memory opt-ins succeed (< 0: all)
int g_export_pixels = 0;             // test builds: most pixels per chain-export launch (0: the product's limit)
#endif

bool cuda_ok(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    snprintf(g_cuda_err, sizeof g_cuda_err, "%s: %s", what, cudaGetErrorString(e));
    (void)cudaGetLastError();  // clear the sticky-free error state
    return false;
}
#define CK(call) do { if (!cuda_ok((call), #call)) return SHFLBW_ERR_CUDA; } while (0)

// A tuning aid: the number that the environment gives at this moment, kUnset without one.  Read where it is asked for (50 ns), so that
// no pointer into the environment, which another thread may change, is kept.
constexpr int kUnset = INT_MIN;
int tuned(const char* name) { const char* e = getenv(name); return e ? atoi(e) : kUnset; }

// Every kernel of this library is launched with the programmatic-stream-serialization attribute:
// it may start while the previous kernel of the stream drains, sets itself up (barriers, TMEM,
// item table), and only then waits for that kernel's completion (griddepcontrol.wait in the
// kernels).  Stream order of all data accesses is unchanged.  SHFLBW_PDL=0 turns it off.
bool use_pdl() {
    static const bool on = [] { const char* e = getenv("SHFLBW_PDL"); return !(e && atoi(e) == 0); }();
    return on;
}
template <typename... Params, typename... Args>
cudaError_t launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = use_pdl() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

int ensure_buffer(void** buf, size_t* have, size_t need) {
    if (*have >= need && *buf) return SHFLBW_OK;
    if (*buf) { cudaFree(*buf); *buf = nullptr; *have = 0; }
    CK(cudaMalloc(buf, need));
    *have = need;
    return SHFLBW_OK;
}

// The device copy lives on the GPU that was current in shflbw_matrix_to_device; launching its
// pointers on another GPU would fault, so ops insist on that GPU being current.
bool on_current_device(const shflbw_matrix& m) {
    int dev = -1;
    return m.d_meta && cudaGetDevice(&dev) == cudaSuccess && dev == m.device;
}

// Conv scratch grows without freeing the outgrown buffer: states initialised earlier keep
// non-owning pointers to it.  Everything is released with the matrix's device copy.
int grow_scratch(shflbw_matrix& m, void** buf, size_t* have, size_t need) {
    if (*have >= need && *buf) return SHFLBW_OK;
    void* fresh = nullptr;
    CK(cudaMalloc(&fresh, need));
    if (*buf) m.retired.push_back(*buf);
    *buf = fresh;
    *have = need;
    return SHFLBW_OK;
}

// Streams and events of the pipelined host-buffer calls, owned by the handle (made on first use).
int host_pipeline(shflbw_matrix* m, cudaStream_t* s_in, cudaStream_t* s_k, cudaStream_t* s_out,
                         cudaEvent_t** e_in, cudaEvent_t** e_k) {
    if (!m->host_streams[0]) {
        for (int i = 0; i < 3; ++i) {
            cudaStream_t st_ = nullptr;
            CK(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
            m->host_streams[i] = st_;
        }
        for (int i = 0; i < 16; ++i) {
            cudaEvent_t ev_ = nullptr;
            CK(cudaEventCreateWithFlags(&ev_, cudaEventDisableTiming));
            m->host_events[i] = ev_;
        }
    }
    *s_in = (cudaStream_t)m->host_streams[0]; *s_k = (cudaStream_t)m->host_streams[1];
    *s_out = (cudaStream_t)m->host_streams[2];
    *e_in = (cudaEvent_t*)&m->host_events[0]; *e_k = (cudaEvent_t*)&m->host_events[8];
    return SHFLBW_OK;
}

// ---- kernel table -------------------------------------------------------------------
using PanelKernel = void (*)(const shflbw::PanelParams);
struct PanelChoice { PanelKernel fn; size_t smem; int tokens; int stages; int pw; int threads; int variant; int gather; };

template <int V, int TM, int KS, int STAGES, int PW, int MODE, int GROUPS = 2, int GATHER = shflbw::kGatherCpAsync,
          int EW = 8, bool BIAS = false, bool ADDEND = false, int SLOTS = 0>
PanelChoice choice() {
    using Cfg = shflbw::PanelCfg<V, TM, KS, STAGES, PW, MODE, GROUPS, GATHER, EW, ADDEND, SLOTS>;
    return {shflbw::panel_umma_kernel<V, TM, KS, STAGES, PW, MODE, GROUPS, GATHER, EW, BIAS, ADDEND, SLOTS>, (size_t)Cfg::SMEM_BYTES, Cfg::T,
            STAGES, PW, Cfg::THREADS, 0, GATHER};
}

// TMA tensor map of a dense operand (`rows` rows of `cols` fp16, `pitch` bytes from one to the next; rows may
// overlap): box = 64 tokens x 1 row (what one row of a tile::gather4 fetches), 128-byte swizzle (the layout
// tcgen05.mma reads), zero fill outside the tensor.  The driver entry point is looked up once.
int encode_map(const void* base, long long rows, long long cols, long long pitch, unsigned long long out[16]) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode enc = nullptr;
    if (!enc) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr));
        if (!fn || qr != cudaDriverEntryPointSuccess) return SHFLBW_ERR_CUDA;
        enc = (Encode)fn;
    }
    static_assert(sizeof(CUtensorMap) == 128, "tensor map size");
    alignas(64) CUtensorMap tm;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {64, 1}, estr[2] = {1, 1};
    const CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_cuda_err, sizeof g_cuda_err, "cuTensorMapEncodeTiled failed: %d", (int)r);
        return SHFLBW_ERR_CUDA;
    }
    std::memcpy(out, &tm, 128);
    return SHFLBW_OK;
}

// Pipeline shape per (V, tile): non-zero columns per stage (KS) and ring depth (as many stages
// as fit beside the 16 KB of epilogue tiles).
// Shapes of the TMA gather: four stages at a time, by two warps each, SpMM with rows in lanes by four: its items are
// deep and its epilogue fits the 80 registers that 25 warps leave (4096^3 V = 64 26.7 -> 25.3 us, V = 128 21.2 -> 20.2,
// 4096x4096x1024 density 0.5 24.8 -> 23.1; with tokens in lanes 11008x4096x512 V = 32 32.7 -> 33.3).
template <int V, int TM, int STAGES, int MODE, bool BIAS>
PanelChoice regular(int gather) {
    constexpr int PW = MODE == shflbw::kPanelSpmmRows ? 16 : 8;
    constexpr bool SPMM = MODE == shflbw::kPanelSpmm || MODE == shflbw::kPanelSpmmRows;
    if constexpr (!(SPMM && BIAS && TM == 2))                // (spmm_gather)
        if (gather == shflbw::kGatherCpAsync) return choice<V, TM, 64, STAGES, 8, MODE, 2, shflbw::kGatherCpAsync, 8, BIAS>();
    return choice<V, TM, 64, STAGES, PW, MODE, 4, shflbw::kGatherTma, 8, BIAS>();
}
template <int MODE, bool BIAS = false>
bool lookup(int V, int tile, PanelChoice* out, int gather = shflbw::kGatherCpAsync, int wide_ring = 0, int wide_pw = 3, bool box = false) {
    if constexpr (MODE == shflbw::kPanelConvChain) {
        if (box) {                                           // box epilogue (see the kernel)
            if (gather != shflbw::kGatherTma || !wide_ring || tile != 256 || V != 64) return false;
            *out = choice<64, 2, 32, 6, 3, MODE, 3, shflbw::kGatherTma, 16, false, false, 3>();
            return true;
        }
    }
    if constexpr (MODE == shflbw::kPanelSpmm || MODE == shflbw::kPanelConvChain) {
        // Shallow items (at most 64 non-zero columns): sixteen epilogue warps and three producer
        // warps, each a group of its own (20 warps: 96 registers per thread); stages of 32 columns,
        // six of them beside the 32 KB of epilogue tiles and the 64 KB of addend slots, so that up to
        // six items' inputs are in flight from HBM (five: 37.5 -> 40.5 us on 14x14x256 -> 1024 at batch
        // 256, the rest equal); eight in the instance without the slots.  Built for 64-row blocks.
        // wide_ring: 6 or 8 stages, 0 for the regular kernels.
        // Three gather warps with a stage each at a time, whichever the gather: with two of them the TMA issue was the
        // longest of an item's steps from 32 columns on (chained 14x14x256 -> 1024 with residual, batch 256, 102
        // columns a block: 57.2 us, three 47.0, three by cp.async 49.9; 28x28x256 -> 512 without residual, batch
        // 128, 48 columns: 36.8, 30.0, 33.1).  With a residual and up to 48 columns two: the addends are what such a layer
        // waits for, and fetching the stages ahead of them faster only gets in their way (in the network, batch 118, three
        // and two: 56x56x64 -> 256, 10 columns, 87.6 and 78.4 us; 28x28x128 -> 512, 20, 48.6 and 45.2; 14x14x256 -> 1024,
        // 40, 30.8 and 29.6; 7x7x512 -> 2048, 80, 22.5 both; without residual 56x56x64 -> 256 48.1 and 54.4), unless the
        // output is beyond 256 MB, where HBM decides (batch 256: 28x28x128 -> 512, 206 MB, 90.7 and 79.9; 56x56x64 -> 256,
        // 411 MB, 183 and 202).  set_residual chooses.
        if (wide_ring && tile == 256 && V == 64) {
            if (gather == shflbw::kGatherTma) {
                if constexpr (MODE == shflbw::kPanelConvChain)
                    if (wide_ring == 6 && wide_pw == 2) { *out = choice<64, 2, 32, 6, 2, MODE, 2, shflbw::kGatherTma, 16, BIAS, true>(); return true; }
                *out = wide_ring == 8 ? choice<64, 2, 32, 8, 3, MODE, 3, shflbw::kGatherTma, 16, BIAS, false>()
                                      : choice<64, 2, 32, 6, 3, MODE, 3, shflbw::kGatherTma, 16, BIAS, true>();
                return true;
            }
            if constexpr (MODE == shflbw::kPanelConvChain) {
                *out = wide_ring == 8 ? choice<64, 2, 32, 8, 3, MODE, 3, shflbw::kGatherCpAsync, 16, BIAS, false>()
                                      : choice<64, 2, 32, 6, 3, MODE, 3, shflbw::kGatherCpAsync, 16, BIAS, true>();
                return true;
            }
            return false;
        }
    }
    if constexpr (MODE == shflbw::kPanelSpmmRows || MODE == shflbw::kPanelConvChainRows) {   // rows in TMEM lanes: V must be a legal UMMA M
        switch (V * 1000 + tile) {
            case 64128:  *out = regular<64, 1, 8, MODE, BIAS>(gather); return true;
            case 64256:  *out = regular<64, 2, 5, MODE, BIAS>(gather); return true;
            case 128128: *out = regular<128, 1, 6, MODE, BIAS>(gather); return true;
            case 128256: *out = regular<128, 2, 4, MODE, BIAS>(gather); return true;
            default: return false;
        }
    } else {
        if constexpr (MODE == shflbw::kPanelSpmm || MODE == shflbw::kPanelConv || MODE == shflbw::kPanelConvScatter) {
            // 16-row blocks: UMMA N = 16, one or two 128-token accumulators per item (18 / 34 KB stages)
            if (V == 16 && tile == 128) { *out = regular<16, 1, 8, MODE, BIAS>(gather); return true; }
            if (V == 16 && tile == 256) { *out = regular<16, 2, 5, MODE, BIAS>(gather); return true; }
        }
        switch (V * 1000 + tile) {
            case 32128:  *out = regular<32, 1, 8, MODE, BIAS>(gather); return true;    // 20 KB stages
            case 32256:  *out = regular<32, 2, 5, MODE, BIAS>(gather); return true;    // 36 KB
            case 64128:  *out = regular<64, 1, 8, MODE, BIAS>(gather); return true;    // 24 KB
            case 64256:  *out = regular<64, 2, 5, MODE, BIAS>(gather); return true;    // 40 KB
            default: break;
        }
        if (V == 128 && tile == 128) { *out = regular<128, 1, 6, MODE, BIAS>(gather); return true; }   // 32 KB
        if (V == 128 && tile == 256) { *out = regular<128, 2, 4, MODE, BIAS>(gather); return true; }   // 48 KB
        return false;
    }
}

// Persistent launch: one CTA per SM, more only when a CTA's share would overflow its item table.
unsigned persistent_grid(int num_items, int sms) {
    int g = num_items < sms ? num_items : sms;
    const int need = (num_items + shflbw::kPanelMaxItemsPerCta - 1) / shflbw::kPanelMaxItemsPerCta;
    return (unsigned)(g > need ? g : need);
}

constexpr int kMaxDevices = 64;

// SM count of the current device, looked up once per device.
int sm_count() {
    static int cached[kMaxDevices] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev >= 0 && dev < kMaxDevices && cached[dev] > 0) return cached[dev];
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (dev >= 0 && dev < kMaxDevices) cached[dev] = n;
    return n;
}

// How a convolution counts its tokens when it gathers by TMA: a box is 64 consecutive tokens, and has to be 128
// consecutive bytes of the staged input.  Without a halo (Wp == Wo) all tokens of an image plane are; with one
// those of an output row, which then counts as so many pixels (a multiple of 64 tokens); with a stride those of one
// pixel.  Returns the pixels that a row counts as, 0 where boxes do not fit.
int tma_row_pix(int Wo, int Wp, int Bp, int stride) {
    if (stride == 1 && Wp == Wo) return Wo;
    int pixels = 1;                                           // that make up whole boxes
    while (pixels * Bp % 64) pixels *= 2;
    return stride > 1 && pixels > 1 ? 0 : (Wo + pixels - 1) / pixels * pixels;
}

// SHFLBW_GATHER=0 takes the cp.async gather everywhere, 1 has an SpMM gather by TMA where it would not by itself
// (tuning aids).  Asked for when a state is made.
bool tma_wanted() { const int e = tuned("SHFLBW_GATHER"); return e == kUnset || e == 1; }

// The gather of an SpMM: TMA, unless rows share 32-byte sectors (8 or 24 tokens), there are few of them, and many blocks
// want each.  The SMs then fetch the same few lines of L2 over and over, and the copy engine's requests to one line queue
// up, the more so where a block takes neighbouring rows.  By TMA and by cp.async, 8 tokens, density 0.5: K = 256, 700
// blocks of 16 rows 15.3 and 8.6 us; K = 768, 148 of 16 9.9 and 5.8; K = 1024, 344 of 64 19.1 and 12.5; K = 2360, 94 of
// 32 14.9 and 9.6; K = 4000, 375 of 32 34.0 and 36.2.  Below 0.4: K = 1024, 688 of 16 at 0.25 19.5 and 11.8; K = 1272,
// 175 of 16 at 0.39 8.4 and 8.8; K = 512, 148 of 16 at 0.1 3.9 and 4.0; a stage of 16 columns, K = 128, 362 of 16 4.7 and
// 5.2.  24 tokens, K = 256, 700 of 32 at 0.5 18.4 and 9.8, 192 of 16 at 0.4 5.0 and 5.0; 40, K = 144, 313 of 32 5.4 and
// 5.2; 16, whose rows are whole sectors, K = 1024, 688 of 16 at 0.25 8.2 and 11.8.
// With a bias 256-token tiles are built for the TMA gather only, without one the other is there to compare with
// (SHFLBW_GATHER=0).
int spmm_gather(long long K, int N, int row_blocks, long long padded_cols, int tile, bool with_bias) {
    if (tile == 256 && with_bias) return shflbw::kGatherTma;
    if (const int e = tuned("SHFLBW_GATHER"); e != kUnset) return e == 1 ? shflbw::kGatherTma : shflbw::kGatherCpAsync;
    const bool dense = 20 * padded_cols > 9 * K * row_blocks;
    const bool crowded = padded_cols > 16ll * row_blocks && ((N == 8 && padded_cols >= 40 * K && K <= (dense ? 3072 : 1024)) ||
                                                             (N == 24 && padded_cols >= 150 * K && K <= 341));
    return crowded && tile == 128 ? shflbw::kGatherCpAsync : shflbw::kGatherTma;
}

// Whether the rows of the blocks lie in the TMEM lanes (SpMM, and SpConv that writes planes): `pays`, or what SHFLBW_SWAP=0|1
// forces (tuning aid).
bool rows_in_lanes(int V, bool pays) {
    if (V != 64 && V != 128) return false;
    const int e = tuned("SHFLBW_SWAP");
    return e == kUnset ? pays : e != 0;
}
bool is_deep(long long padded_cols, int row_blocks) { return padded_cols >= 192ll * row_blocks; }

// Token tile: a persistent CTA works through ceil(items / SMs) items in turn; an item of 128 tokens takes about 2/3 of
// the time of one of 256 (half the gathered bytes, the same number of pipeline stages; eight rounds of SpMM items, K =
// 2048, density 0.2, by TMA: V = 16 0.66, 32 0.66, 64 0.63, 128 0.65; by cp.async 0.68 to 0.78).  256 halves the
// value-panel traffic per token and is the default; 128 where the dense extent is too small to give every SM a few items.
// SHFLBW_TILE=128|256 overrides (tuning aid).
long long rounds_of_items(long long n_tokens, int tile, int row_blocks) {
    const int sms = sm_count() > 0 ? sm_count() : 148;
    return ((n_tokens + tile - 1) / tile * row_blocks + sms - 1) / sms;
}
int pick_tile(long long n_tokens, int row_blocks) {
    if (const int e = tuned("SHFLBW_TILE"); e == 128 || e == 256) return e;
    return n_tokens <= 128 || rounds_of_items(n_tokens, 128, row_blocks) * 2 < rounds_of_items(n_tokens, 256, row_blocks) * 3 ? 128 : 256;
}

// The tile of an SpMM: also 128 tokens where that takes three quarters of the time's rounds (two of 256 or three of 128 for 1.0 to
// 1.5 items per SM), from 100 columns a block on, at 128 rows from 48; and five sixths (three or five rounds) at 128 rows from 64
// columns and at up to 32 rows from 200.  Below, an item is mostly epilogue, of which two tiles have more.  256 and 128 tokens, us:
//   2944x1504x1752, V = 128, 246 columns 11.4 and 9.4; 9536x1256x232, V = 64, 116: 7.5 and 6.3; 5504x2744x152, V = 32, 496: 10.4 and 9.0;
//   400x2312x1872, V = 16, 219: 6.3 and 5.9; 3712x280x1520, V = 128, 56: 6.9 and 5.9; 832x400x1520, V = 32, 39: 4.7 and 4.8;
//   five sixths: 8576x728x1096, V = 128, 99: 15.5 and 14.0; 976x2488x1184, V = 16, 562: 13.2 and 12.3; 2912x352x416, V = 16, 123: 6.4 and 6.5;
//   896x520x5536, V = 64, 182: 7.9 and 8.2.  Over 70 shapes on the 128 side 7 % less.
// 16 rows and rows of B that are not whole sectors (N % 16 = 8; every second one is fetched in five sectors per box instead of four, so
// that the gather is more of an item): the 128-token side also where it saves fewer rounds.  128 over 256 tokens, means of 835 shapes by
// rounds of 128 for one of 256 (up to 1.67 / 1.75 / 1.8 / 11:6 / 1.9): from 200 columns on 0.93 / 0.95 / 0.96 / 0.95 / 0.97, with C
// 0.93 / 0.96 / 0.97 / 0.99 / 1.00; 165 to 199 columns 0.92 / 0.96 / 0.98 / 0.99 / 1.01; these with C, whose second epilogue a steady run of
// rounds does not hide, up to seven rounds of 256 tokens 0.95 / 0.98 / 0.99 / 1.00 / 1.04, from eight on 0.99 / 1.02 / 1.08 / 1.12 / 1.09
// (4096x3200x1400, 165 columns, 20 and 11 rounds: 20.3 and 24.3 us).  Below, with C, 1.1 to 1.2 from 1.75 on; whole sectors:
// 3072x768x1024, 192 columns 10.9 and 12.0; 32 rows 0.96 to 1.04, with C 1.04 to 1.25.
int spmm_tile(int V, long long N, int row_blocks, long long padded_cols, bool with_c) {
    const int tile = pick_tile(N, row_blocks);
    if (tile == 128 || tuned("SHFLBW_TILE") != kUnset) return tile;
    const long long r1 = rounds_of_items(N, 128, row_blocks), r2 = rounds_of_items(N, 256, row_blocks);
    if (r1 * 4 <= r2 * 6 && padded_cols >= (V == 128 ? 48ll : 100ll) * row_blocks) return 128;
    if (V == 16 && N % 16 && (padded_cols >= 200ll * row_blocks ? r1 * 20 <= r2 * 38
                                                                 : padded_cols >= 170ll * row_blocks && r1 * 6 <= r2 * 11 && !(with_c && r2 > 7)))
        return 128;
    return r1 * 6 <= r2 * 10 && V != 64 && padded_cols >= (V == 128 ? 64ll : 200ll) * row_blocks ? 128 : 256;
}

// The gather of a convolution, and the pixels that an output row counts as.  TMA, unless the padding of the rows
// costs more time in rounds of items (those of the tile that each side takes) than the gather saves: a stage takes it
// about 650 clk and the cp.async gather 870 to 1000.  cp.async and TMA in us:
//   Rounds of one tile: up to a quarter more of them (14x14x512 -> 2048, batch 16, V = 64, 3 -> 4 rounds: 28.0 and 28.6; V
// = 32, 6 -> 7: 35.9 and 33.5; 13x13x256 -> 2048, batch 24, V = 64, 900 columns a block, 4 -> 5: 42.7 and 41.7); a fifth for
// taller blocks with tokens in lanes and one or two stages of columns, whose items are more epilogue than gather
// (17x17x256, batch 24: chained -> 1024, V = 64, 102 columns, 4 -> 5: 12.7 and 14.1; -> 2048 in NHWC, V = 128, 40 columns:
// 27.1 and 28.9; less than half a stage, chained 19x19x56 -> 320, batch 79, V = 64, 4 -> 5: 9.6 and 8.4).  Where there are
// more of them the tokens count, too: at most 1.3 times as many (chained 17x17x952 -> 512, batch 51, V = 64, 4 -> 5 rounds of
// 1.41 times the tokens: 67.6 and 71.5; 12x12x16 -> 1088, batch 50, V = 32, 8 -> 10, 1.33: 12.9 and 13.9; no more rounds,
// 17x17x776 -> 608, batch 1, V = 32, 2 -> 2, 1.41: 44.6 and 34.9).
//   Padding that takes one or two rounds of 128-token items to as many of 256: only for blocks of up to a stage of
// columns (V = 32, 40 columns: 9.45 and 8.95, 54: 4.3 and 3.9, 100: 4.0 and 4.6; V = 64 chained, 40: 4.07 and 3.99, 64: 4.4
// and 4.6, 300: 5.5 and 6.3; V = 128, 40: 10.2 and 10.9, 300: 12.9 and 15.7).
//   128 rows with tokens in lanes write the longest items of all.  Into NHWC, padding that fills the chip leaves no SM to
// the passes around (10x10x24 -> 1792, batch 6, 98 -> 140 items: 10.0 and 11.3); deep ones (is_deep) gain as much from the gather (38 shapes
// of 207 to 870 columns whose padding does so, TMA over cp.async 0.89 to 1.06, mean 0.98).  Chained, with a stage of columns and part of
// a second one, whose few copies the TMA gather's longer way to the first bytes does not repay, they gather by cp.async
// (28x28x256 -> 256, 3x3, batch 64, 100 columns 12.2 and 12.1 without and 15.6 and 15.7 with a residual; 14x14x1024 -> 512,
// batch 32, 6.4 and 7.0, 7.5 and 7.8; batch 8, 28x28x256 -> 256, 4.9 and 5.2), and up to three stages where there are fewer
// items than SMs or the rows are padded (27x27x256 -> 256, 3x3, batch 100, 157 columns, with residual: 34.1 and 36.1).  Otherwise TMA: 16 columns 10.9 and 10.1, 48 14.4 and 13.1 with a residual, 200 13.8 and 12.9, 800 29.5 and
// 26.2, 2000 59.8 and 49.3 (28x28x256 -> 256, batch 64).
struct ConvTokens { int row_pix; int gather; };
ConvTokens conv_tokens(int Ho, int Wo, int Wp, int Bp, int stride, int V, int row_blocks, long long padded_cols, bool chain) {
    const ConvTokens plain{Wo, shflbw::kGatherCpAsync};
    const int row_pix = tma_wanted() ? tma_row_pix(Wo, Wp, Bp, stride) : 0;
    const long long before = (long long)Ho * Wo * Bp, after = (long long)Ho * row_pix * Bp;
    if (!row_pix || after >= (1ll << 31)) return plain;
    const int tile0 = pick_tile(before, row_blocks), tile1 = pick_tile(after, row_blocks);
    const long long rounds0 = rounds_of_items(before, tile0, row_blocks), rounds1 = rounds_of_items(after, tile1, row_blocks);
    const long long cost0 = rounds0 * (tile0 == 128 ? 2 : 3), cost1 = rounds1 * (tile1 == 128 ? 2 : 3);
    if (V == 128 && !is_deep(padded_cols, row_blocks)) {
        const bool few = (after + tile1 - 1) / tile1 * row_blocks <= (sm_count() > 0 ? sm_count() : 148);
        if (chain && (few || row_pix != Wo ? tile1 == 256 || padded_cols > 64ll * row_blocks
                          : padded_cols > 64ll * row_blocks && padded_cols <= 128ll * row_blocks)) return plain;
        if (!chain && 4 * after > 5 * before && rounds1 == 1 && 10 * ((after + tile1 - 1) / tile1 * row_blocks) > 9ll * (sm_count() > 0 ? sm_count() : 148))
            return plain;
    }
    const bool short_items = tile1 > tile0 && V <= 64 && padded_cols <= (V == 64 && chain ? 48ll : 64ll) * row_blocks;
    const bool tight = V >= 64 && padded_cols > 32ll * row_blocks && padded_cols <= 128ll * row_blocks;
    const bool roomy = cost1 <= cost0 || padded_cols <= 32ll * row_blocks || 10 * after <= 13 * before;
    const bool pays = short_items || (roomy && (tight ? 5 * cost1 <= 6 * cost0 : 4 * cost1 <= 5 * cost0));
    return pays ? ConvTokens{row_pix, shflbw::kGatherTma} : plain;
}

// Opt a kernel in to its dynamic shared memory once per (device, kernel): the host-buffer
// calls initialise an op per chunk, and the attribute call is not free.
int allow_smem(const void* fn, size_t bytes) {
    static shflbw::OncePerDevice done;
    int dev = 0;
    CK(cudaGetDevice(&dev));
#ifdef SHFLBW_FAULT_INJECT
    if (g_set_ups_left == 0) return SHFLBW_ERR_CUDA;
    if (g_set_ups_left > 0) --g_set_ups_left;
#endif
    return done.run(fn, dev, [&]() -> int {
        CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        return SHFLBW_OK;
    });
}
int allow_smem(PanelKernel fn, size_t bytes) { return allow_smem((const void*)fn, bytes); }

// The kernel of a plan, allowed its shared memory.  wide_ring: sixteen epilogue warps and that many stages (lookup), 0: eight.
template <int MODE>
int pick_panel(int V, int tile, bool rows, int wide_ring, int gather, PanelChoice* out) {
    if constexpr (MODE == shflbw::kPanelSpmm) { if (wide_ring) gather = shflbw::kGatherTma; }   // (built for it only)
    bool found;
    if (rows)
        found = MODE == shflbw::kPanelSpmm ? lookup<shflbw::kPanelSpmmRows>(V, tile, out, gather) : lookup<shflbw::kPanelConvChainRows>(V, tile, out, gather);
    else
        found = lookup<MODE>(V, tile, out, gather, wide_ring);
    if (!found) return SHFLBW_ERR_UNSUPPORTED;
    out->variant = rows ? 1 : wide_ring ? 2 : 0;
    if (wide_ring == 8) {                    // a residual may be bound to the state later on
        PanelChoice with_addend;
        if (!lookup<MODE>(V, tile, &with_addend, gather, 6)) return SHFLBW_ERR_UNSUPPORTED;
        const int rc = allow_smem(with_addend.fn, with_addend.smem);
        if (rc != SHFLBW_OK) return rc;
    }
    return allow_smem(out->fn, out->smem);
}

// Sixteen epilogue warps, tokens in lanes: SHFLBW_EPILOGUE_WARPS=8|16 forces the choice (tuning aid).
bool wide_wanted(int V, int tile, bool pays) {
    if (V != 64 || tile != 256) return false;
    const int e = tuned("SHFLBW_EPILOGUE_WARPS");
    return e == kUnset ? pays : e == 16;
}
// Their ring: eight stages where nothing is added and a block takes two stages, which a ring of six holds for
// three items only (28x28x128 -> 512, batch 256, no residual, 40 columns: 56.6 us with six, 54.7 with eight); blocks
// of one stage are as fast with six (26 columns: 48.5, with eight 49.7).
int wide_ring_of(bool addend, long long padded_cols, int row_blocks) { return !addend && padded_cols > 32ll * row_blocks ? 8 : 6; }

// Whether an SpMM runs with sixteen epilogue warps (tokens in lanes).  Few columns a block and several items per SM: an item is
// all epilogue.  V = 64, N = 4096, 6.9 items per SM, eight warps / sixteen / rows in lanes: 16 columns 13.8 / 11.1 / 11.5 us, 64 15.1 /
// 12.4 / 12.8, 80 15.4 / 13.1 / 13.3, 100 16.0 / 13.9 / 13.8, 128 16.8 / 15.5 / 14.7; with fewer items rows in lanes win (three: 48
// columns 8.2 / 7.6 / 7.2).  Rows of B and D that are no whole 32-byte sectors (N % 16 = 8), where rows in lanes store 16 bytes
// at a time: N = 4104, 16 columns 15.0 / 11.9 / 16.2, 80 17.4 / 15.4 / 19.3, 100 18.0 / 17.1 / 20.2, 128 19.0 / 19.3 / 21.3; N = 2056,
// 3.8 items per SM, 16 / 48 / 90 columns 9.0 and 7.9 / 9.8 and 8.6 / 11.0 and 10.2.  `sectors`: whole ones.  With C: N = 4096, 16 columns 18.0 / 14.7 / 33.1,
// 160 23.3 / 19.4 / 38.2; two items per SM, 16 / 48 / 90 columns 7.3 and 6.7 / 7.6 and 7.4 / 8.7 and 8.0; 1.35: 6.2 and 5.6 / 6.3 and
// 6.6 / 8.0 and 7.2.
bool spmm_wide(int V, int tile, int N, bool sectors, bool with_c, long long padded_cols, int row_blocks) {
    const long long items = (N + 255) / 256 * (long long)row_blocks, sms = sm_count() > 0 ? sm_count() : 148;
    const int most = with_c ? 160 : sectors ? 80 : 104;
    return wide_wanted(V, tile, padded_cols <= (long long)most * row_blocks && (with_c ? items >= 2 * sms : sectors ? items >= 4 * sms : 2 * items >= 7 * sms));
}
// Whether its rows lie in the TMEM lanes where it does not.  They store 32 bytes a lane if D's rows are whole sectors: then
// always (V = 64, 1024x1024x64, 16 / 96 / 256 columns, tokens and rows: 2.93 and 2.71 / 3.67 and 3.26 / 4.27 and 3.69;
// 512x1024x16384 8.9 and 7.6 / 10.4 and 9.3 / 12.5 and 11.7; 4096x1024x4096, 256: 19.1 and 19.2; V = 128 13.9 and 11.2 / 16.1 and
// 13.3 / 18.6 and 16.7).  If not, up to 64 tokens (4096x1024x40, 40 / 120 / 400 columns: 3.13 and 2.88 / 3.97 and 3.49 / 5.48 and
// 4.73), and 64 rows in 128-token tiles from a stage and a half on (1024x4096x504: 3.31 and 3.41 / 4.11 and 4.09 / 5.62 and
// 5.39), not beyond (4096x1024x3000, 120 / 400: 15.0 and 16.8 / 26.9 and 30.3; V = 128 14.1 and 15.5 / 21.4 and 22.6).  C is read
// after the accumulator there, which pays for 64 rows from 1600 columns on (4096x4096x4096, 400 / 1600 / 3200: 31.4 and 45.6 /
// 76.6 and 76.8 / 137 and 128; V = 128 33.1 and 49.5 / 59.0 and 65.2 / 102 and 103), and on 24 tokens or fewer, of which C has
// little, from three stages on (8 tokens: 448x3704, V = 64, 977 columns 6.56 and 5.90, 8704x2312, V = 128, 187 columns 4.60 and
// 4.24; 40 tokens, 4096x4096, 256 columns 4.70 and 5.03).
bool spmm_rows(int V, int tile, int N, bool sectors, bool with_c, long long padded_cols, int row_blocks) {
    const bool whole = sectors || N <= 64;
    if (with_c) return rows_in_lanes(V, (V == 64 && whole && padded_cols >= 1600ll * row_blocks) || (N <= 24 && is_deep(padded_cols, row_blocks)));
    return rows_in_lanes(V, whole || (V == 64 && tile == 128 && padded_cols >= 96ll * row_blocks));
}

// The same for chained layers, of `tokens` tokens counted with the padding of their rows.  Tokens in lanes, which write (and
// read a residual) in runs of 64 bytes a row where rows in lanes scatter 16 bytes a lane, up to the depth where the MMA is
// what an item waits for: at 64 rows two of 48 clk instead of one of 80 for the 256 tokens; at 128 rows it is 128 clk
// either way.  Tokens and rows, us: V = 64, 28x28x256 -> 256, 3x3, batch 64: 256 columns 16.6 and 20.6 (with residual 20.7 and
// 28.3), 800 35.4 and 36.9, 1200 49.0 and 48.2 (51.7 and 54.5), 2000 75.8 and 70.7 (78.4 and 76.6); 7x7x512 -> 512, batch 8,
// 600 columns 6.2 and 6.3; V = 128: 400 17.1 and 20.9, 2000 49.3 and 48.9 (52.2 and 56.1).
// Layers of fewer than 16 items, and those whose rows are no whole boxes of the TMA gather and go into an output with a halo
// beside them, keep the line at three stages of columns.
bool chain_rows(int V, bool padded_into_halo, long long items, long long padded_cols, int row_blocks) {
    const bool deep = is_deep(padded_cols, row_blocks);
    return rows_in_lanes(V, deep && (padded_into_halo || items < 16 || (V == 64 && padded_cols >= 1200ll * row_blocks)));
}
// At most 64 non-zero columns per block, and two or three items per SM (eight and sixteen, 13 / 40 / 60 columns: 2.7 items
// 7.25 and 6.62 / 7.54 and 7.57 / 7.79 and 7.73, 3.6 8.6 and 7.6 / 9.1 and 8.8 / 9.2 and 9.0; 1.7 5.76 and 5.57 / 6.14 and 6.33 /
// 6.32 and 6.33; 28x28x256 -> 256, batch 128, 64 columns 19.2 and 17.9, 96 21.3 and 21.1, 128 21.9 and 23.0).
bool chain_wide(int V, int tile, long long items, long long padded_cols, int row_blocks) {
    return wide_wanted(V, tile, padded_cols <= 64ll * row_blocks && 2 * items >= 5ll * (sm_count() > 0 ? sm_count() : 148));
}

// Argument and range checks shared by every NHWC SpConv entry point.  The kernels index the
// staged input with 32-bit element offsets and the output with 32-bit offsets whose all-ones
// value is a sentinel, so both extents are bounded here, before anything is launched.
struct ConvShape { int Ho, Wo, Bp; long long tokens, staged_elems; };
int check_conv_call(const shflbw_matrix* f, int B, int Hin, int Win, int stride, const void* ifmap,
                    const void* ofmap, ConvShape* cs) {
    if (!f || !ifmap || !ofmap || B <= 0 || Hin <= 0 || Win <= 0 || stride <= 0) return SHFLBW_ERR_INVALID_ARG;
    if (!f->is_filter) return SHFLBW_ERR_INVALID_ARG;
    if (!on_current_device(*f)) return SHFLBW_ERR_NOT_ON_DEVICE;
    if (f->C % 8 || f->R > 255 || f->S > 255) return SHFLBW_ERR_UNSUPPORTED;
    if (((uintptr_t)ifmap | (uintptr_t)ofmap) & 15) return SHFLBW_ERR_UNSUPPORTED;
    if (B > (1 << 24) || Hin > (1 << 24) || Win > (1 << 24)) return SHFLBW_ERR_UNSUPPORTED;   // keeps the products below in 64 bits
    cs->Ho = (Hin + stride - 1) / stride; cs->Wo = (Win + stride - 1) / stride;
    cs->Bp = (B + 7) / 8 * 8;
    cs->tokens = (long long)cs->Ho * cs->Wo * cs->Bp;
    const long long plane = (long long)(Hin + f->R - 1) * (Win + f->S - 1);        // < 2^50
    if (plane >= (1ll << 31) || cs->tokens >= (1ll << 31)) return SHFLBW_ERR_UNSUPPORTED;
    cs->staged_elems = plane * cs->Bp;                                              // < 2^56
    if (cs->staged_elems >= (1ll << 31) || cs->staged_elems * f->C >= (1ll << 31)) return SHFLBW_ERR_UNSUPPORTED;
    cs->staged_elems *= f->C;
    if ((long long)B * cs->Ho * cs->Wo >= (1ll << 32) || (long long)B * cs->Ho * cs->Wo * f->F >= (1ll << 32) - 1)
        return SHFLBW_ERR_UNSUPPORTED;                                              // 32-bit output offsets
    return SHFLBW_OK;
}

int check_kernel_arg(int kernel) {
    return (kernel == SHFLBW_KERNEL_AUTO || kernel == SHFLBW_KERNEL_TCGEN05 || kernel == SHFLBW_KERNEL_SIMT)
               ? SHFLBW_OK : SHFLBW_ERR_INVALID_ARG;
}

}  // namespace

// Scratch of shflbw_spconv_exec_static_scratch: part of the library image, present on every
// GPU that loads the library.  In HOST code this name is only a handle for
// cudaGetSymbolAddress -- it is not a device address and must never be handed to a kernel.
static __device__ __align__(256) unsigned char g_static_scratch[SHFLBW_STATIC_SCRATCH_BYTES];

namespace {
void* g_static_scratch_addr[kMaxDevices] = {};  // device address of the array, per device
}  // namespace

namespace shflbw {
void drop_device_copy(shflbw_matrix& m) {
    void** bufs[] = {&m.d_meta, &m.d_val, &m.stage_in, &m.stage_c, &m.stage_out, &m.conv_in, &m.conv_out};
    for (void** b : bufs) if (*b) { cudaFree(*b); *b = nullptr; }
    for (void* r : m.retired) cudaFree(r);
    m.retired.clear();
    for (void*& st : m.host_streams) if (st) { cudaStreamDestroy((cudaStream_t)st); st = nullptr; }
    for (void*& ev : m.host_events) if (ev) { cudaEventDestroy((cudaEvent_t)ev); ev = nullptr; }
    m.stage_in_bytes = m.stage_c_bytes = m.stage_out_bytes = m.conv_in_bytes = m.conv_out_bytes = 0;
    m.d_kptr = m.d_kidx = m.d_perm = m.d_kcrs = nullptr;
    m.d_status = nullptr;
    m.device = -1;
}
}  // namespace shflbw

namespace {
// Whether a linear layer on a few tokens goes to the one-launch kernel: where its blocks, of 8 tokens each, are few and read little.
// Their registers (40 to 56 a thread) let four to six blocks of 256 threads be on an SM at once, shared memory often fewer, and the
// limit is four; up to 8 tokens it is what shared memory lets in, eight at most, in two waves (66 shapes of 4 to 8 blocks an SM: 0.22 to 0.68
// of the two launches' device time).  Device time, two launches and one: 4096 x 4096, V = 64, density 0.1 on 1 / 8 / 16 / 37 / 64 tokens
// 5.4 / 5.7 / 5.1 / 5.5 / 5.4 and 2.9 / 3.4 / 4.1 / 5.0 / 9.2 us (64: 3.5 blocks an SM, of which 3 are resident); the host gains another
// 2.2 us.  Over 160 shapes the two are equal near 270 KB an SM, of value panels and of the 32-byte sectors of x, less 20 KB for
// every further pass over a block's columns (3712 x 7816, density 0.086, 18 tokens, 242 KB in two passes: 6.4 and 7.5;
// 4096 x 4096 on 37 tokens: 245 KB in one), and from five blocks an SM on (1104 x 368, V = 16, 81 tokens: 4.6 and 5.5).  Up to 8 tokens
// the panel kernel is no faster with so few (8608 x 440, V = 16, 3 tokens: 7.2 and 3.4): as far as 400 KB (9344 x 5224, V = 128, 5 tokens,
// 319 KB in three passes: 8.9 and 7.4; 2304 x 4440, V = 128, 3 tokens, 382 KB in three: 8.4 and 8.3).
bool linear_direct_pays(const shflbw_matrix& m, int tokens, int N, size_t smem) {
    if (const int e = tuned("SHFLBW_LINEAR_DIRECT"); e != kUnset) return e != 0;
    const long long sms = sm_count() > 0 ? sm_count() : 148, row_blocks = m.nrow / m.brow, blocks = row_blocks * (N / shflbw::kDirectTokens);
    const long long resident = 228 * 1024 / ((long long)smem + 1024) < 8 ? 228 * 1024 / ((long long)smem + 1024) : 8;
    const bool few = N == shflbw::kDirectTokens;
    if (m.kptr.empty() || blocks > sms * (few || resident < 4 ? resident : 4)) return false;
    const long long panels = m.kptr.back() * 2ll * m.brow, cols = m.kptr.back() / row_blocks;
    const long long row = 2ll * m.ncol < 32 * cols ? 2ll * m.ncol : 32 * cols;           // bytes that a block reads of a token
    const long long all = panels * (N / shflbw::kDirectTokens) + row_blocks * tokens * row;
    const long long per_sm = all / (blocks < sms ? blocks : sms), passes = (m.max_cols + shflbw::kDirectCols - 1) / shflbw::kDirectCols;
    return per_sm + 20 * 1024 * (passes - 1) <= (few ? 400 : 256) * 1024;
}
}  // namespace

extern "C" {

const char* shflbw_last_cuda_error(void) { return g_cuda_err; }

int shflbw_set_wait_limit_cycles(long long cycles) {
    if (cycles < 1000) return SHFLBW_ERR_INVALID_ARG;
    g_wait_limit = cycles;
    return SHFLBW_OK;
}

#ifdef SHFLBW_FAULT_INJECT
// Test builds only: launches issued after this call run with one producer warp withholding its
// barrier arrivals from stage `stage` on (< 0: off), so that the consumer's bounded wait gives up.
int shflbw_debug_withhold_arrivals_from(int stage) { g_inject_from = stage; return SHFLBW_OK; }
// ... and after this call `n` kernels are allowed their shared memory, the next ones refused (n < 0: off).
int shflbw_debug_fail_set_up_after(int n) { g_set_ups_left = n; return SHFLBW_OK; }
#endif

int shflbw_matrix_to_device(shflbw_matrix_t* m) {
    if (!m) return SHFLBW_ERR_INVALID_ARG;
    if (m->d_meta) return SHFLBW_OK;
    int rc = shflbw::validate(*m);
    if (rc != SHFLBW_OK) return rc;
    shflbw::build_host_images(*m);
    int dev = 0;
    CK(cudaGetDevice(&dev));
    auto up8 = [](size_t v) { return (v + 7) / 8 * 8; };
    const size_t o_ptr = 0, o_idx = up8(m->kptr.size()), o_perm = o_idx + up8(m->kidx.size()),
                 o_crs = o_perm + up8(m->row_permute_ids.size()), o_stat = o_crs + up8(m->kcrs.size()),
                 total = o_stat + 8;
    std::vector<int> img(total, 0);
    std::copy(m->kptr.begin(), m->kptr.end(), img.begin() + o_ptr);
    std::copy(m->kidx.begin(), m->kidx.end(), img.begin() + o_idx);
    std::copy(m->row_permute_ids.begin(), m->row_permute_ids.end(), img.begin() + o_perm);
    std::copy(m->kcrs.begin(), m->kcrs.end(), img.begin() + o_crs);
    CK(cudaMalloc(&m->d_meta, total * sizeof(int)));
    if (!cuda_ok(cudaMalloc(&m->d_val, (m->kval.size() + m->kval_logical.size()) * 2), "cudaMalloc(values)")) {
        cudaFree(m->d_meta); m->d_meta = nullptr;
        return SHFLBW_ERR_CUDA;
    }
    CK(cudaMemcpy(m->d_meta, img.data(), total * sizeof(int), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(m->d_val, m->kval.data(), m->kval.size() * 2, cudaMemcpyHostToDevice));
    if (!m->kval_logical.empty())
        CK(cudaMemcpy((uint16_t*)m->d_val + m->kval.size(), m->kval_logical.data(), m->kval_logical.size() * 2, cudaMemcpyHostToDevice));
    const int* base = (const int*)m->d_meta;
    m->d_kptr = base + o_ptr;
    m->d_kidx = base + o_idx;
    m->d_perm = m->row_permute ? base + o_perm : nullptr;
    m->d_kcrs = m->kcrs.empty() ? nullptr : base + o_crs;
    m->d_status = (int*)m->d_meta + o_stat;
    m->device = dev;
    return SHFLBW_OK;
}

int shflbw_matrix_on_device(const shflbw_matrix_t* m) { return m && m->d_meta ? 1 : 0; }

int shflbw_matrix_device_status(const shflbw_matrix_t* m) {
    if (!m || !m->d_status) return SHFLBW_ERR_NOT_ON_DEVICE;
    int word = 0;
    CK(cudaDeviceSynchronize());
    CK(cudaMemcpy(&word, m->d_status, sizeof word, cudaMemcpyDeviceToHost));
    if (word != 0) {
        CK(cudaMemset(m->d_status, 0, sizeof word));
        snprintf(g_cuda_err, sizeof g_cuda_err, "device status word = %d", word);
        return SHFLBW_ERR_DEVICE_TIMEOUT;
    }
    return SHFLBW_OK;
}

// Callers hold these states by value: their sizes belong to the version that shflbw_abi_version() gives, and a new field to a
// new one (or into bytes that are there).
static_assert(sizeof(shflbw_spmm_state_t) == 304 && sizeof(shflbw_spconv_state_t) == 232, "layout of ABI version 1");

// ------------------------------------------------------------------------------ SpMM --

static int plan_spmm(const shflbw_matrix_t* m, int N, const void* B, float alpha, const void* C,
                     float beta, void* D, int kernel, bool with_bias, shflbw_spmm_state_t* out) {
    if (!out) return SHFLBW_ERR_INVALID_ARG;
    std::memset(out, 0, sizeof *out);
    if (!m || !B || !D || N <= 0) return SHFLBW_ERR_INVALID_ARG;
    if (check_kernel_arg(kernel) != SHFLBW_OK) return SHFLBW_ERR_INVALID_ARG;
    if (beta != 0.f && !C) return SHFLBW_ERR_INVALID_ARG;
    if (!on_current_device(*m)) return SHFLBW_ERR_NOT_ON_DEVICE;  // reference: assert(device_synced)
    // The reference asserts bcol == 1 here (spmm/blockwise_op.h:86); the kernel image lists the
    // bcol columns of a block one by one, so wider blocks run on the same kernels.
    // Row-block heights 16/32/64/128 (what the reference instantiates, spmm/blockwise_library.cu:15-31)
    // run on the tensor-core kernel.
    if (kernel != SHFLBW_KERNEL_SIMT && m->brow != 16 && m->brow != 32 && m->brow != 64 && m->brow != 128)
        return SHFLBW_ERR_UNSUPPORTED;
    if (kernel == SHFLBW_KERNEL_SIMT && (N + 127) / 128 > 65535) return SHFLBW_ERR_UNSUPPORTED;   // column tiles ride in grid.y
    if (N % 8) return SHFLBW_ERR_UNSUPPORTED;                   // 16-byte rows of fp16
    const uintptr_t al = (uintptr_t)B | (uintptr_t)D | (uintptr_t)C;
    if (al & 15) return SHFLBW_ERR_UNSUPPORTED;
    if ((long long)m->nrow * N >= (1ll << 32) || (long long)m->ncol * N >= (1ll << 40))
        return SHFLBW_ERR_UNSUPPORTED;                          // 32-bit element offsets into C / D

    out->M = m->nrow; out->N = N; out->K = m->ncol; out->V = m->brow;
    out->num_row_blocks = m->nrow / m->brow;
    out->alpha = alpha; out->beta = beta;
    out->B = B; out->C = C; out->D = D;
    out->blk_ptr = m->d_kptr; out->blk_idx = m->d_kidx; out->blk_val = m->d_val;
    out->perm = m->d_perm; out->status_word = m->d_status;
    if (kernel == SHFLBW_KERNEL_SIMT) {
        out->kernel = SHFLBW_KERNEL_SIMT;
        out->block_x = 128; out->grid_x = m->nrow; out->grid_y = (N + 127) / 128;   // rows in grid.x: no 65535 limit
        out->tokens_per_cta = 128; out->stages = 0; out->shared_mem_size = 0;
    } else {
        PanelChoice ch;
        const long long padded_cols = m->kptr.empty() ? 0 : m->kptr.back();
        const int blocks = out->num_row_blocks, tile = spmm_tile(m->brow, N, blocks, padded_cols, beta != 0.f);
        const bool sectors = N % 16 == 0 && !((uintptr_t)D & 31);
        const int swap = tuned("SHFLBW_SWAP");
        const bool wide = (swap == kUnset || swap == 0) && spmm_wide(m->brow, tile, N, sectors, beta != 0.f, padded_cols, blocks);
        const bool rows = !wide && spmm_rows(m->brow, tile, N, sectors, beta != 0.f, padded_cols, blocks);
        const int ring = wide ? wide_ring_of(beta != 0.f, padded_cols, blocks) : 0;
        int rc = pick_panel<shflbw::kPanelSpmm>(m->brow, tile, rows, ring, spmm_gather(m->ncol, N, blocks, padded_cols, tile, with_bias), &ch);
        if (rc != SHFLBW_OK) return rc;
        out->kernel = SHFLBW_KERNEL_TCGEN05;
        out->tokens_per_cta = ch.tokens; out->stages = ch.stages; out->producer_warps = ch.pw; out->variant = ch.variant;
        out->gather = ch.gather;
        if (ch.gather == shflbw::kGatherTma) {
            if ((rc = encode_map(B, m->ncol, N, 2ll * N, out->tmap_b)) != SHFLBW_OK) return rc;
            out->tmap_of = B; out->tmap_cols = N; out->tmap_rows = m->ncol;
        }
        out->tiles_n = (N + ch.tokens - 1) / ch.tokens;
        out->num_items = out->tiles_n * out->num_row_blocks;
        const int sms = sm_count();
        if (sms <= 0) return SHFLBW_ERR_CUDA;
        out->block_x = ch.threads;
        out->grid_x = persistent_grid(out->num_items, sms); out->grid_y = 1;
        out->shared_mem_size = ch.smem;
    }
    out->init_success = 1;
    return SHFLBW_OK;
}

int shflbw_spmm_init(const shflbw_matrix_t* m, int N, const void* B, float alpha, const void* C,
                     float beta, void* D, int kernel, shflbw_spmm_state_t* out) {
    return plan_spmm(m, N, B, alpha, C, beta, D, kernel, false, out);
}

// The panel kernel of an initialised SpMM state, allowed its shared memory.  The state is a POD and may have
// been copied: the function pointer is re-derived from the recorded configuration.  bias: the instance that
// adds a bias (init allowed the one without).
static int spmm_panel(const shflbw_spmm_state_t* st, bool bias, PanelChoice* ch) {
    const int wide_ring = st->variant != 2 ? 0 : st->beta != 0.f ? 6 : st->stages;   // (an addend needs its slots)
    const bool found =
        bias ? st->variant == 1 ? lookup<shflbw::kPanelSpmmRows, true>(st->V, st->tokens_per_cta, ch, st->gather)
                                : lookup<shflbw::kPanelSpmm, true>(st->V, st->tokens_per_cta, ch, st->gather, wide_ring)
             : st->variant == 1 ? lookup<shflbw::kPanelSpmmRows>(st->V, st->tokens_per_cta, ch, st->gather)
                                : lookup<shflbw::kPanelSpmm>(st->V, st->tokens_per_cta, ch, st->gather, wide_ring);
    if (!found || ch->gather != st->gather) return SHFLBW_ERR_INVALID_ARG;
    return bias ? allow_smem(ch->fn, ch->smem) : SHFLBW_OK;
}

// bias: nullptr, or one value per output row, added to the fp16 product (state without C).
static int launch_spmm_panel(const shflbw_spmm_state_t* st, const PanelChoice& ch, const void* bias, cudaStream_t s) {
    shflbw::PanelParams p{};
    p.blk_ptr = st->blk_ptr; p.blk_idx = st->blk_idx; p.blk_val = (const __half*)st->blk_val;
    p.perm = st->perm; p.status_word = st->status_word; p.alpha = st->alpha; p.beta = st->beta;
    p.wait_limit = g_wait_limit; p.inject_from = g_inject_from; p.idx_limit = (unsigned)(st->K - 1);
    p.B = (const __half*)st->B; p.C = (const __half*)st->C; p.D = (__half*)st->D; p.N = st->N;
    if (bias) { p.C = (const __half*)bias; p.beta = 1.f; }
    p.wide_stores = (st->N % 16 == 0) && (((uintptr_t)st->D & 31) == 0);
    // The state is the caller's: an operand that they exchanged is gathered through a map of its own.
    if (st->gather == shflbw::kGatherTma) {
        if (st->tmap_of == st->B && st->tmap_cols == st->N && st->tmap_rows == st->K) {
            std::memcpy(p.tmap_b, st->tmap_b, sizeof p.tmap_b);
        } else {
            const int rc = encode_map(st->B, st->K, st->N, 2ll * st->N, p.tmap_b);
            if (rc != SHFLBW_OK) return rc;
        }
    }
    p.num_items = st->num_items; p.tiles_n = st->tiles_n;
    p.div_tiles = shflbw::make_fast_div(st->tiles_n); p.div_bp = p.div_row = shflbw::make_fast_div(1);
    // Tile-major item order: concurrent CTAs gather from the same few token tiles of B (SHFLBW_ITEM_ORDER=0|1
    // forces block-major / tile-major; tuning aid).
    p.num_blocks = st->num_row_blocks; p.div_blocks = shflbw::make_fast_div(st->num_row_blocks);
    p.tile_major = 1;
    if (const int e = tuned("SHFLBW_ITEM_ORDER"); e != kUnset) p.tile_major = e != 0;
    CK(launch(ch.fn, dim3(st->grid_x, st->grid_y), dim3(ch.threads), ch.smem, s, p));
    CK(cudaGetLastError());
    return SHFLBW_OK;
}

int shflbw_spmm_exec(const shflbw_spmm_state_t* st, void* stream) {
    if (!st || !st->init_success) return SHFLBW_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (st->kernel == SHFLBW_KERNEL_SIMT) {
        shflbw::simt_spmm<<<dim3(st->grid_x, st->grid_y), st->block_x, 0, s>>>(
            st->blk_ptr, st->blk_idx, (const __half*)st->blk_val, st->perm, (const __half*)st->B,
            (const __half*)st->C, (__half*)st->D, st->M, st->N, st->V, st->alpha, st->beta);
        CK(cudaGetLastError());
        return SHFLBW_OK;
    }
    PanelChoice ch;
    const int rc = spmm_panel(st, false, &ch);
    return rc != SHFLBW_OK ? rc : launch_spmm_panel(st, ch, nullptr, s);
}

int shflbw_linear_exec(const shflbw_matrix_t* m, int tokens, const void* x, const void* bias, void* xt, int N, void* out,
                       void* stream) {
    if (!m || !xt || !out || N <= 0 || tokens > N || (x && tokens <= 0)) return SHFLBW_ERR_INVALID_ARG;
    if (((uintptr_t)x | (uintptr_t)bias) & 1) return SHFLBW_ERR_UNSUPPORTED;
    shflbw_spmm_state_t st;
    int rc = plan_spmm(m, N, xt, 1.f, nullptr, 0.f, out, SHFLBW_KERNEL_AUTO, bias != nullptr, &st);   // (asks for 16-byte aligned xt, out and N % 8)
    if (rc != SHFLBW_OK) return rc;
    PanelChoice ch;                                          // all set-up comes before the first launch
    if ((rc = spmm_panel(&st, bias != nullptr, &ch)) != SHFLBW_OK) return rc;
    if (x) {
        const long long tiles = (long long)((m->ncol + 63) / 64) * ((N + 63) / 64);   // < 2^31: ncol * N < 2^40 or refused above
        if (tiles >= (1ll << 31)) return SHFLBW_ERR_UNSUPPORTED;
        CK(launch(shflbw::transpose_tokens, dim3((unsigned)tiles), dim3(256), 0, (cudaStream_t)stream, (const __half*)x, (__half*)xt, tokens,
                  m->ncol, N, (int)(m->ncol % 8 == 0 && ((uintptr_t)x & 15) == 0)));
    }
    return launch_spmm_panel(&st, ch, bias, (cudaStream_t)stream);
}

int shflbw_linear_direct(const shflbw_matrix_t* m, int tokens, const void* x, const void* bias, int N, void* out, void* stream) {
    if (!m || !x || !out || N <= 0 || tokens <= 0 || tokens > N) return SHFLBW_ERR_INVALID_ARG;
    if (((((uintptr_t)x | (uintptr_t)bias) & 1) | ((uintptr_t)out & 15)) || N % 8) return SHFLBW_ERR_UNSUPPORTED;
    if (!on_current_device(*m)) return SHFLBW_ERR_NOT_ON_DEVICE;
    if ((long long)m->nrow * N >= (1ll << 32) || (long long)m->ncol * N >= (1ll << 40)) return SHFLBW_ERR_UNSUPPORTED;   // as shflbw_spmm_init
    void (*fn)(const shflbw::DirectParams);
    shflbw::DirectParams p{};
    switch (m->brow) {
        case 16: fn = shflbw::linear_direct<16>; break;
        case 32: fn = shflbw::linear_direct<32>; break;
        case 64: fn = shflbw::linear_direct<64>; break;
        case 128: fn = shflbw::linear_direct<128>; break;
        default: return SHFLBW_ERR_UNSUPPORTED;
    }
    const size_t smem = shflbw::direct_smem(m->brow, m->max_cols);
    if (!linear_direct_pays(*m, tokens, N, smem)) return SHFLBW_ERR_UNSUPPORTED;
    const int rc = allow_smem((const void*)fn, shflbw::direct_smem(m->brow, shflbw::kDirectCols));
    if (rc != SHFLBW_OK) return rc;
    p.blk_ptr = m->d_kptr; p.blk_idx = m->d_kidx; p.perm = m->d_perm; p.blk_val = (const __half*)m->d_val;
    p.x = (const __half*)x; p.bias = (const __half*)bias; p.out = (__half*)out;
    p.tokens = tokens; p.K = m->ncol; p.N = N; p.groups = N / shflbw::kDirectTokens;
    CK(launch(fn, dim3((unsigned)(m->nrow / m->brow * p.groups)), dim3(256), smem, (cudaStream_t)stream, p));
    return SHFLBW_OK;
}

int shflbw_spmm_launches_per_exec(const shflbw_spmm_state_t* st) { return st && st->init_success ? 1 : 0; }

// Host-buffer SpMM.  The dense operand is cut into column chunks that move through three
// streams -- host-to-device copy of chunk i+1, kernel on chunk i, device-to-host copy of chunk
// i-1 -- so that on a full-duplex link the call costs about the larger of the two transfers
// instead of their sum plus the kernel.  (Overlap needs page-locked host buffers; pageable ones
// work, the copies then serialise.)  A chunk is staged contiguously ([K][w] / [M][w]) by a strided
// 2-D copy, so the kernels run unchanged on dense chunks.
// mode 0: the real call.  1: the same copies through the same streams and events, no kernel
// (what the link alone costs).  2: as 1, but every chunk moves as one contiguous block of the
// same size (what the strided form of the chunk copies costs on top).
static int spmm_host_impl(shflbw_matrix_t* m, int N, const void* B_host, float alpha, const void* C_host,
                          float beta, void* D_host, int mode) {
    if (!m || !B_host || !D_host || N <= 0) return SHFLBW_ERR_INVALID_ARG;
    if (beta != 0.f && !C_host) return SHFLBW_ERR_INVALID_ARG;
    if (N % 8) return SHFLBW_ERR_UNSUPPORTED;
    int rc = shflbw_matrix_to_device(m);
    if (rc != SHFLBW_OK) return rc;
    // Before any staging buffer or stream is made: they would belong to the wrong GPU.
    if (!on_current_device(*m)) return SHFLBW_ERR_NOT_ON_DEVICE;
    const size_t bB = (size_t)m->ncol * N * 2, bD = (size_t)m->nrow * N * 2;
    if ((rc = ensure_buffer(&m->stage_in, &m->stage_in_bytes, bB)) != SHFLBW_OK) return rc;
    if ((rc = ensure_buffer(&m->stage_out, &m->stage_out_bytes, bD)) != SHFLBW_OK) return rc;
    if (beta != 0.f && (rc = ensure_buffer(&m->stage_c, &m->stage_c_bytes, bD)) != SHFLBW_OK) return rc;

    // chunk width: a quarter of N rounded up to whole 256-token tiles; narrow operands go in one piece
    int w = N;
    int want = 4;
    if (const int e = tuned("SHFLBW_HOST_CHUNKS"); e > 0 && e <= 8) want = e;
    if (N >= 2048 && want > 1) w = ((N + want - 1) / want + 255) / 256 * 256;
    const int chunks = (N + w - 1) / w;
    constexpr int kMaxChunks = 8;
    if (chunks > kMaxChunks) return SHFLBW_ERR_UNSUPPORTED;   // cannot happen: w >= N/4

    // streams and events live in the handle (creating and destroying them costs more than the
    // overlap gains on a call of about a millisecond)
    auto fail = [&](int code) { cudaDeviceSynchronize(); return code; };
#define CKH(call) do { if (!cuda_ok((call), #call)) return fail(SHFLBW_ERR_CUDA); } while (0)
    cudaStream_t s_in, s_k, s_out;
    cudaEvent_t *e_in, *e_k;
    if ((rc = host_pipeline(m, &s_in, &s_k, &s_out, &e_in, &e_k)) != SHFLBW_OK) return rc;
    const size_t pitch_h = (size_t)N * 2;
    for (int i = 0; i < chunks; ++i) {
        const int c0 = i * w, wi = (N - c0 < w) ? N - c0 : w;
        // chunk i of the staging buffers: contiguous [rows][wi] blocks, one after the other
        __half* dB = (__half*)m->stage_in + (size_t)m->ncol * c0;
        __half* dD = (__half*)m->stage_out + (size_t)m->nrow * c0;
        __half* dC = beta != 0.f ? (__half*)m->stage_c + (size_t)m->nrow * c0 : nullptr;
        if (mode == 2)
            CKH(cudaMemcpyAsync(dB, (const __half*)B_host + (size_t)m->ncol * c0, (size_t)wi * 2 * m->ncol,
                                cudaMemcpyHostToDevice, s_in));
        else
        CKH(cudaMemcpy2DAsync(dB, (size_t)wi * 2, (const __half*)B_host + c0, pitch_h, (size_t)wi * 2, m->ncol,
                              cudaMemcpyHostToDevice, s_in));
        if (dC)
            CKH(cudaMemcpy2DAsync(dC, (size_t)wi * 2, (const __half*)C_host + c0, pitch_h, (size_t)wi * 2, m->nrow,
                                  cudaMemcpyHostToDevice, s_in));
        CKH(cudaEventRecord(e_in[i], s_in));
        CKH(cudaStreamWaitEvent(s_k, e_in[i], 0));
        if (mode == 0) {
            shflbw_spmm_state_t st;
            rc = shflbw_spmm_init(m, wi, dB, alpha, dC, beta, dD, SHFLBW_KERNEL_AUTO, &st);
            if (rc == SHFLBW_OK) rc = shflbw_spmm_exec(&st, s_k);
            if (rc != SHFLBW_OK) return fail(rc);
        }
        CKH(cudaEventRecord(e_k[i], s_k));
        CKH(cudaStreamWaitEvent(s_out, e_k[i], 0));
        if (mode == 2)
            CKH(cudaMemcpyAsync((__half*)D_host + (size_t)m->nrow * c0, dD, (size_t)wi * 2 * m->nrow,
                                cudaMemcpyDeviceToHost, s_out));
        else
        CKH(cudaMemcpy2DAsync((__half*)D_host + c0, pitch_h, dD, (size_t)wi * 2, (size_t)wi * 2, m->nrow,
                              cudaMemcpyDeviceToHost, s_out));
    }
    CKH(cudaStreamSynchronize(s_out));
    CKH(cudaStreamSynchronize(s_k));
    CKH(cudaStreamSynchronize(s_in));
#undef CKH
    return SHFLBW_OK;
}

int shflbw_spmm_host(shflbw_matrix_t* m, int N, const void* B_host, float alpha, const void* C_host,
                     float beta, void* D_host) {
    return spmm_host_impl(m, N, B_host, alpha, C_host, beta, D_host, 0);
}

int shflbw_spmm_host_copies_only(shflbw_matrix_t* m, int N, const void* B_host, void* D_host, int contiguous) {
    return spmm_host_impl(m, N, B_host, 1.0f, nullptr, 0.0f, D_host, contiguous ? 2 : 1);
}

// ---------------------------------------------------------------------------- SpConv --

// Shared memory that a relayout of so many blocks asks for on top of its tile, so that an SM holds no more than its
// even share of them (up to seven; eight fit by their threads).  The blocks of a call that follows another are
// resident early, on the SMs that the kernel before leaves first, and wait there: without a limit they pile up on
// those few, which then move everything (24x16x16x160 -> 1856, V = 64, 1x1, unpermuted, calls back to back: 17.3 us;
// with the limit 14.3).  With less than one block per SM the share is one where the kernel before is likely to be
// a panel kernel, as it is behind a call that ends with one (10x27x27x176 -> 624: 13.5 us without, 9.5 with), and
// without a limit behind a last pass, whose blocks are short and everywhere and leave no room for blocks of half an
// SM (4x20x26x96 -> 1312: 16.7 us with, 16.0 without).
constexpr size_t kRelayoutTile = (size_t)shflbw::kRelayoutC * shflbw::kRelayoutSlots * 2;
static size_t relayout_smem(long long blocks, bool has_last_pass) {
    const int sms = sm_count() > 0 ? sm_count() : 148;
    const long long per_sm = (blocks + sms - 1) / sms;
    if (per_sm > 7 || (per_sm == 1 && has_last_pass)) return 0;
    return (size_t)(per_sm == 1 ? 227 : 228 / per_sm - 1) * 1024 - kRelayoutTile;   // of 228 KB, 1 KB a block is the system's
}

#ifdef SHFLBW_FAULT_INJECT
// The bytes of shared memory that a relayout of `blocks` blocks occupies per block.
int shflbw_debug_relayout_smem(long long blocks, int has_last_pass) { return (int)(kRelayoutTile + relayout_smem(blocks, has_last_pass != 0)); }
#endif

// NHWC -> [C][Hin+R-1][Win+S-1][Bp] with a zero halo (origin at (R/2, S/2)); step > 1 (1x1 filters): only the
// pixels that the stride visits, [C][ceil(Hin/step)][ceil(Win/step)][Bp].
// Returns the number of blocks per SM.
static long long launch_relayout(const __half* in, __half* staged, int B, int Bp, int Hin, int Win, int C, int R, int S,
                            cudaStream_t s, int step = 1, bool has_last_pass = true) {
    const int Hp = step > 1 ? (Hin + step - 1) / step : Hin + R - 1, Wp = step > 1 ? (Win + step - 1) / step : Win + S - 1;
    const int PP = Hp * Wp;
    const int NT = Bp < 32 ? Bp : 32, PT = shflbw::kRelayoutSlots / NT;
    const int n_tiles = (Bp + NT - 1) / NT;
    dim3 grid((unsigned)(((PP + PT - 1) / PT) * n_tiles), (unsigned)((C + shflbw::kRelayoutC - 1) / shflbw::kRelayoutC));
    const auto kernel = step > 1 ? shflbw::relayout_nhwc_to_chwn<true> : shflbw::relayout_nhwc_to_chwn<false>;
    const long long blocks = (long long)grid.x * grid.y;
    size_t smem = relayout_smem(blocks, has_last_pass);
    if (smem && allow_smem((const void*)kernel, relayout_smem(1, false)) != SHFLBW_OK) smem = 0;   // only a matter of speed
    (void)launch(kernel, grid, dim3(256), smem, s, in, staged, B, Bp, Hin, Win, Hp, Wp, R / 2, S / 2, C, step);
    const int sms = sm_count() > 0 ? sm_count() : 148;
    return (blocks + sms - 1) / sms;
}

// Dynamic shared memory of unpermute_filters: 16-bit permutation + one F-vector of fp16 per position.
static size_t unperm_smem_bytes(int F) {
    return (size_t)F * 2 * (1 + shflbw::kUnpermThreads / shflbw::unperm_threads_per_pos(F));
}

// Blocks per 64 channels of a chain export: two to eight 64-token steps per block where that leaves several
// blocks per SM, so that a block's scan of the permutation and its start-up are shared.
static long long export_blocks(long long tiles, int F) {
    const int fb = (F + 63) / 64;
    long long gx = (148 * 16 + fb - 1) / fb;
    if (gx < (tiles + 7) / 8) gx = (tiles + 7) / 8;
    return gx < tiles ? gx : tiles;
}

// Chain buffer -> NHWC (see the kernel).
static cudaError_t launch_export(const void* planes, void* out, const int* perm, int Bn, int Bp, int H, int W,
                                         int Hp, int Wp, int ph, int pw, int F, cudaStream_t s) {
    int per = (1 << 30) / Bp > 0 ? (1 << 30) / Bp : 1;                  // pixels per launch: the kernel counts its tokens in 31 bits
#ifdef SHFLBW_FAULT_INJECT
    if (g_export_pixels > 0) per = g_export_pixels;
#endif
    const long long npix = (long long)H * W;
    for (long long pix0 = 0; pix0 < npix; pix0 += per) {
        const int n = (int)(npix - pix0 < per ? npix - pix0 : per);
        const long long tiles = ((long long)n * Bp + 63) / 64;
        const cudaError_t e = launch(shflbw::export_planes_nhwc, dim3((unsigned)export_blocks(tiles, F), (unsigned)((F + 63) / 64)), dim3(256), 0, s, (const __half*)planes,
                                     (__half*)out, perm, Bn, Bp, (int)pix0, n, (int)npix, W, Wp, ph, pw, (size_t)Hp * Wp * Bp, F,
                                     shflbw::make_fast_div(Bp), shflbw::make_fast_div(W));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

#ifdef SHFLBW_FAULT_INJECT
// Chain exports issued after this call cover at most `n` pixels per launch (n <= 0: the product's limit).
int shflbw_debug_set_export_pixels(int n) { g_export_pixels = n; return SHFLBW_OK; }
// The most 64-token steps that a block of a chain export of `tokens` (pixels * padded batch) and F channels takes.
int shflbw_debug_export_steps(long long tokens, int F) {
    const long long tiles = (tokens + 63) / 64, gx = export_blocks(tiles, F);
    return (int)((tiles + gx - 1) / gx);
}
#endif

// What a convolution's tensor maps are of.  Input: one row per pixel that a tap of output pixel (0, 0) reads, `pitch` from
// one to the next, as long as from output pixel (0, 0) to the last: every address that the map allows is inside the
// input.  Output and residual of a chained layer: its planes, up to the last pixel.
struct PlaneMap { const void* base; long long rows, cols, pitch; };
PlaneMap input_map(const shflbw_spconv_state_t& st, const void* base, int Hp, int Wp, int stride) {
    return {base, ((long long)st.C - 1) * Hp * Wp + (long long)(st.R - 1) * Wp + st.S,
            (((long long)st.Ho - 1) * stride * Wp + ((long long)st.Wo - 1) * stride + 1) * st.Bp, 2ll * st.Bp};
}
PlaneMap output_map(const shflbw_spconv_state_t& st, const void* base) {
    const long long OWp = st.Wo + st.out_S - 1, OHp = st.Ho + st.out_R - 1;
    return {base, st.F, ((st.out_R / 2 + st.Ho - 1) * OWp + st.out_S / 2 + st.Wo) * st.Bp, 2 * OHp * OWp * st.Bp};
}
// Whether 64 consecutive tokens of a chained layer are 128 consecutive bytes of an output plane throughout: the rows are
// not padded, and either the output has no halo beside its rows or they are whole boxes.
bool boxes_fit(const shflbw_spconv_state_t& st) {
    return st.row_pix == st.Wo && (st.out_S == 1 || (long long)st.Wo * st.Bp % 64 == 0);
}
// Whether an NHWC call of a permuted filter is computed as planes (below): they leave the panel kernel in runs of 64 bytes,
// the inverse permutation being an address, and the transposing pass reads and writes runs of 128.  Positions out and planes
// out (tokens in lanes), 40 / 110 / 460 columns a block: 14x14x512 -> 2048, 3x3, batch 16, V = 64 17.6 and 15.7 / 18.6 and 16.7 /
// 26.6 and 24.5; 14x14x256 -> 1024 15.4 and 12.1 / 16.8 and 13.5 / 21.3 and 18.0; 56x56x64 -> 64, batch 32 20.4 and 17.7 /
// 21.7 and 19.4 / 27.8 and 24.6; V = 128 12 to 22 % less.  Not where the planes carry an eighth more images than there are
// (28x28x256 -> 512, batch 1, 160 columns: 12.6 and 13.3), with less than an item of 256 tokens per SM (17x17x512 -> 256, 1x1,
// batch 24, 74 columns: 12.1 and 13.4; 14x14x256 -> 512, batch 8, 460: 10.8 and 11.1) at 64 rows (at 128 from half an
// item on: 14 shapes 4 to 12 % less, 31x31x336 -> 640, 1x1 at stride 2, batch 23, 152 columns 16.1 and 13.7), nor for less than a stage of columns
// with padded rows (not looked at).  An unpermuted filter's positions need no further pass (28x28x256 -> 256, 1x1, batch 64,
// 64 columns: 20.7, as planes 31.4; 14x14x512 -> 2048, 3x3, batch 16, 900: 29.0 and 33.2).
// With filters in lanes (28.3 instead of 24.5 for 14x14x512 -> 2048, 460 columns) only at 64 rows from 1200 columns on, as
// the chained layers (14x14x256 -> 1024, 1800 columns: 33.4, tokens 33.8).
// Nor where planes and output together are beyond the L2's 126 MB and of more than 640 filters: the last pass comes to planes that have
// left it.  Planes over positions, means of 260 shapes by these megabytes, 80 to 100 / 126 / 150 / 200 / more: 64 rows 0.90 / 0.94 / 0.99 /
// 1.00 / 1.02, 128 rows 0.95 / 0.98 / 1.01 / 1.06 / 1.08 (16x60x60 of 1920 filters, 1x1: 1.23); up to 640 filters, whose few
// blocks are written sooner after one another, 0.91 / 0.92 / 0.95 / 0.95 / 0.93.
bool conv_planes(const shflbw_matrix& f, int B, int Bp, int tile, long long items, bool padded_rows, long long padded_cols, int row_blocks,
                 long long planes_and_out) {
    if (f.F > 640 && planes_and_out > 126000000) return false;
    return tile == 256 && (f.brow == 128 || items >= (sm_count() > 0 ? sm_count() : 148)) && 8 * (Bp - B) <= Bp && (padded_cols >= 64ll * row_blocks || !padded_rows);
}
// And whether it is for the number of its filters alone, whatever the padding of the batch, the tile and the SMs with items: the last pass
// of positions loads the permutation in every block and holds an F-vector for each position, and gets slow.  Planes over positions,
// means of 450 shapes with fewer than three items per SM, by filters, planes of up to 1.125 / 1.6 / 2 / 8 times the images: up to 512 filters
// 0.96 / 0.98 / 1.04 / 1.13, 1024 0.95 / 0.97 / 0.98 / 1.09, 1536 0.91 / 0.92 / 0.97 / 1.05, 2304 0.89 / 0.88 / 0.91 / 0.99, more 0.82 / 0.82 / 0.81 / 0.87
// (3x39x11x616 -> 3712, 1x1 at stride 2, 200 columns: 20.5 and 14.1 us; 8x8x8x544 -> 2944, V = 128, 290: 15.7 and 11.7).  From
// three items per SM on 0.97 / 1.05 / 0.99 / 1.19 beyond 2304.
bool conv_planes_by_filters(const shflbw_matrix& f, int B, int Bp, long long items, bool padded_rows, long long padded_cols, int row_blocks) {
    return items < 3ll * (sm_count() > 0 ? sm_count() : 148) && (padded_cols >= 64ll * row_blocks || !padded_rows) &&
           (f.F > 2304 || (f.F > 1024 && Bp <= 2 * B));
}

// Whether the panel kernel itself puts a permuted filter's positions in order, value by value: a pass less (2 us and a launch,
// 2.2 us of the host's time), but every 32-byte sector of an F-vector is written once by each block that has a filter in it, and
// the L2 takes some 80 of such partial sectors a clock.  So for small outputs, by the expected sectors that the busiest SM writes; the
// line rises with the share of the SMs that have items, since the pass is spread over all of them.  Scattered over the pass, means of 500
// shapes of all heights in a graph (eager calls 0.01 to 0.05 less) by sectors, up to 1200 / 1800 / 2400 / 2900 / 3500 / 4600: items on up to a
// quarter of the SMs 0.88 / 0.96 / 1.00 / 1.08 / 1.19 / 1.23; to a half 0.89 / 0.94 / 0.98 / 1.04 / 1.13 / 1.19; to three quarters 0.89 / 0.93 /
// 0.94 / 1.02 / 1.04 / 1.13; to all 0.84 / 0.89 / 0.93 / 0.99 / 0.96 / 1.02; several rounds 0.81 / 0.86 / 0.90 / 0.94 / 0.94 / 1.01.  Among the 331
// shapes that scatter by the line one takes 13 % longer, the others up to 9 in a graph and 2 eagerly.
bool conv_scatters(const shflbw_matrix& f, long long positions, long long items) {
    if (const int e = tuned("SHFLBW_CONV_SCATTER"); e != kUnset) return e != 0;
    const long long sms = sm_count() > 0 ? sm_count() : 148;
    if (8 * items < sms) return false;                       // a few blocks keep the general form (2x12x12x128 -> 128: 6.35 us, 5.9 without the pass)
    const double sectors = f.F / 16.0, chunk = f.brow < 32 ? f.brow : 32;
    const double written = sectors * (1 - std::pow(1 - 1 / sectors, chunk)) * (f.F / chunk) * (double)positions;   // in all
    return written / (double)items * (double)((items + sms - 1) / sms) <= 1500 + 1900 * (items < sms ? (double)items / (double)sms : 1.0);
}

// Launch plan of one NHWC SpConv call, without its scratch pointers: kernel choice, grid, and
// the scratch each side needs.  Two plans exist.
//   positions out   relayout -> panel kernel with tokens in TMEM lanes, writing [position][F] in
//                   stored filter order -> (with a filter permutation across blocks) unpermute_filters; small
//                   outputs in logical order at once (conv_scatters).
//   planes out      relayout -> panel kernel writing the output as planes [F][Ho][Wo][Bp] with plane = LOGICAL
//                   channel (the permutation is the row index of its stores, free) -> planes_to_nhwc
//                   transposes the planes to NHWC.  Used for permuted V = 64 / 128 filters and outputs that
//                   fill the chip (conv_planes), with tokens or, where deep, filters in TMEM lanes.
// SHFLBW_CONV_PLANES=0|1 forces the choice (tuning aid).
int plan_conv(const shflbw_matrix* f, int B, int Hin, int Win, int stride, const void* ifmap, void* ofmap,
              float alpha, int kernel, shflbw_spconv_state_t* out, size_t scratch_limit = ~(size_t)0) {
    std::memset(out, 0, sizeof *out);
    if (check_kernel_arg(kernel) != SHFLBW_OK) return SHFLBW_ERR_INVALID_ARG;
    ConvShape cs;
    int rc = check_conv_call(f, B, Hin, Win, stride, ifmap, ofmap, &cs);
    if (rc != SHFLBW_OK) return rc;
    if (kernel != SHFLBW_KERNEL_SIMT && f->brow != 16 && f->brow != 32 && f->brow != 64 && f->brow != 128)
        return SHFLBW_ERR_UNSUPPORTED;
    const int Ho = cs.Ho, Wo = cs.Wo, Bp = cs.Bp;
    const long long tokens = cs.tokens;

    out->B = B; out->Hin = Hin; out->Win = Win; out->C = f->C; out->F = f->F; out->R = f->R; out->S = f->S;
    out->stride = stride; out->Ho = Ho; out->Wo = Wo; out->V = f->brow; out->Bp = Bp;
    out->alpha = alpha; out->ifmap = ifmap; out->ofmap = ofmap;
    out->blk_ptr = f->d_kptr; out->blk_idx = f->d_kidx; out->blk_val = f->d_val;
    out->perm = f->d_perm; out->status_word = f->d_status;
    if (kernel == SHFLBW_KERNEL_SIMT) {
        if ((f->F + 127) / 128 > 65535) return SHFLBW_ERR_UNSUPPORTED;
        out->kernel = SHFLBW_KERNEL_SIMT;
        out->block_x = 128; out->grid_x = (unsigned)(B * Ho * Wo); out->grid_y = (f->F + 127) / 128;   // positions in grid.x
        out->init_success = 1;
        return SHFLBW_OK;
    }
    // The panel kernel reads decoded column ids (channel in 16 bits, taps in 8 bits each).
    if (!f->d_kcrs) return SHFLBW_ERR_UNSUPPORTED;
    out->blk_idx = f->d_kcrs;
    const int row_blocks = f->F / f->brow;
    const long long padded_cols = f->kptr.empty() ? 0 : f->kptr.back();

    // planes out?
    const bool planes_possible = (f->brow == 64 || f->brow == 128) && f->F / 64 <= 65535 &&
                                 (long long)f->F * tokens < (1ll << 32) - 1 && rows_in_lanes(f->brow, true);
    const int ep = tuned("SHFLBW_CONV_PLANES");
    // the input as the panel kernel sees it: a strided 1x1 filter's pixels are staged side by side
    const bool compact = f->R == 1 && f->S == 1;
    const ConvTokens ct = conv_tokens(Ho, Wo, compact ? Wo : Win + f->S - 1, Bp, compact ? 1 : stride, f->brow, row_blocks, padded_cols, false);
    const long long counted = (long long)Ho * ct.row_pix * Bp;
    const int tile = pick_tile(counted, row_blocks);
    const long long items = (counted + tile - 1) / tile * row_blocks;
    // (planes of up to an eighth more images than positions have: not where a fixed scratch holds only these)
    const bool planes_fit = (size_t)cs.staged_elems * 2 + 256 + (size_t)f->F * (size_t)tokens * 2 + 256 <= scratch_limit;
    // The last pass of permuted positions holds the permutation and an F-vector for each position of a block in shared memory
    // (up to 23 244 filters).  Beyond, planes whatever they cost (the same for all sizes of a layer: no small output goes
    // through the scattering kernel either).
    const bool across = f->row_permute && f->kval_logical.empty();        // filters leave their blocks
    const bool pass_fits = !across || (unperm_smem_bytes(f->F) <= 227 * 1024 && f->F <= 65536);
    const bool padded_rows = ct.row_pix != Wo, small = across && conv_scatters(*f, (long long)B * Ho * Wo, items);
    const bool pays = across && (conv_planes(*f, B, Bp, tile, items, padded_rows, padded_cols, row_blocks, 2ll * (B + Bp) * Ho * Wo * f->F) ||
                                 (!small && conv_planes_by_filters(*f, B, Bp, items, padded_rows, padded_cols, row_blocks)));
    const bool planes = planes_possible && (ep != kUnset ? planes_fit && ep != 0 : !pass_fits || (planes_fit && pays));
    if (!planes && !pass_fits) return SHFLBW_ERR_UNSUPPORTED;
    const bool scatter = !planes && small;
    PanelChoice ch;
    if (planes) {
        const int ring = chain_wide(f->brow, tile, items, padded_cols, row_blocks) ? wide_ring_of(false, padded_cols, row_blocks) : 0;
        out->rows = f->brow == 64 && padded_cols >= 1200ll * row_blocks;
        rc = pick_panel<shflbw::kPanelConvChain>(f->brow, tile, out->rows, out->rows ? 0 : ring, ct.gather, &ch);
        out->wide = !out->rows && ring;
    } else if (scatter) {
        rc = pick_panel<shflbw::kPanelConvScatter>(f->brow, tile, false, 0, ct.gather, &ch);
    } else {
        rc = pick_panel<shflbw::kPanelConv>(f->brow, tile, false, 0, ct.gather, &ch);
    }
    if (rc != SHFLBW_OK) return rc;
    if (planes) {
        out->variant = 1;
        out->staged_out_bytes = (size_t)f->F * (size_t)tokens * 2;
    } else {
        out->variant = 0;
        if (!f->kval_logical.empty()) {
            // Rows in logical order: as an unpermuted filter, no pass behind the kernel (56x56x64 -> 64, 3x3, batch 32, V = 64,
            // 115 columns: as planes 19.3 us, so 14.4; 25 filters of one block, 1x1 and 3x3, V = 16 to 128: 13 to 32 % less).
            out->blk_val = (const uint16_t*)f->d_val + f->kval.size();
            out->perm = nullptr;
        } else if (across && !scatter) {
            out->staged_out_bytes = (size_t)B * Ho * Wo * f->F * 2;
            if (unperm_smem_bytes(f->F) > 48 * 1024)
                for (const void* k : {(const void*)shflbw::unpermute_filters<false>, (const void*)shflbw::unpermute_filters<true>})
                    CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)unperm_smem_bytes(f->F)));
        }
    }
    out->kernel = SHFLBW_KERNEL_TCGEN05;
    out->tokens_per_cta = ch.tokens; out->stages = ch.stages; out->producer_warps = ch.pw;
    out->gather = ch.gather; out->row_pix = ct.row_pix;
    out->tiles_n = (int)((counted + ch.tokens - 1) / ch.tokens);
    out->num_items = out->tiles_n * row_blocks;
    const int sms = sm_count();
    if (sms <= 0) return SHFLBW_ERR_CUDA;
    out->block_x = ch.threads;
    out->grid_x = persistent_grid(out->num_items, sms); out->grid_y = 1;
    out->shared_mem_size = ch.smem;
    out->staged_in_bytes = (size_t)cs.staged_elems * 2;     // the whole image, also where a strided 1x1 filter stages less:
                                                            // callers size and check their scratch by the documented formula
    return SHFLBW_OK;
}

int shflbw_spconv_init(shflbw_matrix_t* f, int B, int Hin, int Win, int stride, const void* ifmap,
                       void* ofmap, float alpha, int kernel, shflbw_spconv_state_t* out) {
    if (!out) return SHFLBW_ERR_INVALID_ARG;
    int rc = plan_conv(f, B, Hin, Win, stride, ifmap, ofmap, alpha, kernel, out);
    if (rc != SHFLBW_OK || out->kernel == SHFLBW_KERNEL_SIMT) return rc;
    // Scratch owned by the filter handle, grown on demand.
    if ((rc = grow_scratch(*f, &f->conv_in, &f->conv_in_bytes, out->staged_in_bytes)) != SHFLBW_OK) return rc;
    out->staged_in = f->conv_in;
    if (out->staged_out_bytes) {
        if ((rc = grow_scratch(*f, &f->conv_out, &f->conv_out_bytes, out->staged_out_bytes)) != SHFLBW_OK) return rc;
        out->staged_out = f->conv_out;
    }
    out->init_success = 1;
    return SHFLBW_OK;
}

int shflbw_spconv_exec(const shflbw_spconv_state_t* st, void* stream) { return shflbw_spconv_exec_bias(st, nullptr, stream); }

int shflbw_spconv_exec_bias(const shflbw_spconv_state_t* st, const void* bias, void* stream) {
    if (!st || !st->init_success) return SHFLBW_ERR_INVALID_ARG;
    if (bias && (st->chain || st->kernel == SHFLBW_KERNEL_SIMT || ((uintptr_t)bias & 15))) return SHFLBW_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    if (st->kernel == SHFLBW_KERNEL_SIMT) {
        shflbw::simt_spconv<<<dim3(st->grid_x, st->grid_y), st->block_x, 0, s>>>(
            st->blk_ptr, st->blk_idx, (const __half*)st->blk_val, st->perm, (const __half*)st->ifmap,
            (__half*)st->ofmap, st->B, st->Hin, st->Win, st->C, st->F, st->R, st->S, st->stride, st->Ho,
            st->Wo, st->V, st->alpha);
        CK(cudaGetLastError());
        return SHFLBW_OK;
    }
    const bool planes = !st->chain && st->variant == 1;     // NHWC call computed as planes, then transposed
    PanelChoice ch;
    const bool scatter = !st->chain && !planes && st->perm && !st->staged_out;   // filters to their places, no later pass
    const bool panel_bias = bias && !planes && !st->staged_out;   // no later pass: the panel kernel's epilogue adds the bias
    const int gather = st->gather;
    // (the state is the caller's: a residual that they took away, or a map that the copies' row ids cannot be read from)
    const bool box = st->chain && st->box_res && st->residual && !((uintptr_t)st->residual_map & 15);
    const bool ok_kernel = scatter               ? lookup<shflbw::kPanelConvScatter>(st->V, st->tokens_per_cta, &ch, gather)
                           : panel_bias          ? lookup<shflbw::kPanelConv, true>(st->V, st->tokens_per_cta, &ch, gather)
                           : (!st->chain && !planes) ? lookup<shflbw::kPanelConv>(st->V, st->tokens_per_cta, &ch, gather)
                           : st->rows              ? lookup<shflbw::kPanelConvChainRows>(st->V, st->tokens_per_cta, &ch, gather)
                                                   : lookup<shflbw::kPanelConvChain>(st->V, st->tokens_per_cta, &ch, gather,
                                                                                      !st->wide ? 0 : st->residual ? 6 : st->stages,
                                                                                      st->producer_warps, box);
    if (!ok_kernel) return SHFLBW_ERR_INVALID_ARG;
    if ((panel_bias && !scatter) || (st->box_res && !box)) {              // (init allowed the other kernel; before anything is launched)
        const int rc = allow_smem(ch.fn, ch.smem);
        if (rc != SHFLBW_OK) return rc;
    }
    // 1. NHWC -> channel-major, batch-innermost staging with a zero halo (chained layers get
    //    their input in that layout already).
    //    A strided 1x1 filter visits 1 / stride^2 of the pixels: only those are staged, as an image of the
    //    output's size that is then read at stride 1 (27x27x256 -> 14x14x512, batch 5: 3.4 -> 2.5 us).
    const int step = !st->chain && st->R == 1 && st->S == 1 ? st->stride : 1;
    const int Hp = step > 1 ? st->Ho : st->Hin + st->R - 1, Wp = step > 1 ? st->Wo : st->Win + st->S - 1;
    shflbw::PanelParams p{};
    p.Xs = (const __half*)(st->chain ? st->ifmap : st->staged_in);
    p.stride = st->stride / step;
    p.row_pix = st->row_pix;
    if (gather == shflbw::kGatherTma) {
        const PlaneMap m = input_map(*st, p.Xs, Hp, Wp, p.stride);
        const int rc = encode_map(m.base, m.rows, m.cols, m.pitch, p.tmap_b);
        if (rc != SHFLBW_OK) return rc;
    }
    long long relayout_per_sm = 0;
    if (!st->chain)
        relayout_per_sm = launch_relayout((const __half*)st->ifmap, (__half*)st->staged_in, st->B, st->Bp, st->Hin, st->Win, st->C,
                                          st->R, st->S, s, step, planes || st->staged_out);
    // 2. implicit-GEMM panel kernel.
    // Where it ends the call: see the kernel.  A call that stages many blocks per SM is likely to be followed by another
    // one, whose first blocks cannot be spread over the SMs (26x48x48x1024 -> 96 at stride 2, back to back: 75.6 us, 78.9
    // with the trigger); it is long enough not to miss the 1 us.
    p.trigger_late = relayout_per_sm <= 7;
    p.blk_ptr = st->blk_ptr; p.blk_idx = st->blk_idx; p.blk_val = (const __half*)st->blk_val;
    p.perm = st->perm; p.status_word = st->status_word; p.alpha = st->alpha; p.beta = 0.f;
    p.wait_limit = g_wait_limit; p.inject_from = g_inject_from;
    p.N = st->Ho * p.row_pix * st->Bp;
    p.out = (__half*)(st->staged_out ? st->staged_out : st->ofmap);
    if (st->chain) {
        p.res = (const __half*)st->residual; p.res_map = st->residual_map;
        const int OHp = st->Ho + st->out_R - 1;
        p.OWp = st->Wo + st->out_S - 1; p.oph = st->out_R / 2; p.opw = st->out_S / 2;
        p.out_plane = OHp * p.OWp * st->Bp; p.relu = st->relu;
        if (box) {
            if (!boxes_fit(*st)) return SHFLBW_ERR_INVALID_ARG;
            const PlaneMap m = output_map(*st, st->residual);
            const int rc = encode_map(m.base, m.rows, m.cols, m.pitch, p.tmap_res);
            if (rc != SHFLBW_OK) return rc;
        }
    } else if (planes) {
        p.OWp = st->Wo; p.oph = 0; p.opw = 0; p.out_plane = st->Ho * st->Wo * st->Bp;
        p.out_logical = 1;                                   // plane index = logical channel
    }
    p.idx_limit = (unsigned)((((long long)st->C - 1) * Hp * Wp + (long long)(st->R - 1) * Wp + (st->S - 1)) * st->Bp);
    p.Bn = st->B; p.Bp = st->Bp; p.Hp = Hp; p.Wp = Wp; p.Cin = st->C; p.F = st->F;
    p.R = st->R; p.S = st->S; p.Ho = st->Ho; p.Wo = st->Wo;
    p.num_items = st->num_items; p.tiles_n = st->tiles_n;
    p.div_tiles = shflbw::make_fast_div(st->tiles_n); p.div_bp = shflbw::make_fast_div(st->Bp); p.div_row = shflbw::make_fast_div(p.row_pix);
    p.num_blocks = st->F / st->V; p.div_blocks = shflbw::make_fast_div(p.num_blocks);
    // Block-major item order for the convolutions: running a token tile's filter blocks at the same time
    // (tile-major) was measured equal on the ResNet-50 stack and on config 3, whose inputs are small next
    // to their outputs (SHFLBW_ITEM_ORDER=1 forces tile-major; tuning aid).
    p.tile_major = 0;
    if (const int e = tuned("SHFLBW_ITEM_ORDER"); e != kUnset) p.tile_major = e != 0;
    if (panel_bias) p.C = (const __half*)bias;
    CK(launch(ch.fn, dim3(st->grid_x, st->grid_y), dim3(ch.threads), ch.smem, s, p));
    // 3. back to NHWC in logical channel order.
    if (planes) {
        const int npix = st->Ho * st->Wo;
        CK(launch(bias ? shflbw::planes_to_nhwc<true> : shflbw::planes_to_nhwc<false>,
                  dim3((unsigned)(((long long)npix * st->Bp + 63) / 64), (unsigned)(st->F / 64)), dim3(256), 0, s,
                  (const __half*)st->staged_out, (__half*)st->ofmap, (const __half*)bias, st->B, st->Bp, npix, st->F));
    } else if (st->staged_out) {
        const int num_pos = st->B * st->Ho * st->Wo;
        const int per_block = shflbw::kUnpermThreads / shflbw::unperm_threads_per_pos(st->F);
        int blocks = (num_pos + per_block - 1) / per_block;
        if (blocks > 148 * 16) blocks = 148 * 16;
        CK(launch(bias ? shflbw::unpermute_filters<true> : shflbw::unpermute_filters<false>, dim3(blocks), dim3(shflbw::kUnpermThreads), unperm_smem_bytes(st->F), s,
                  (const __half*)st->staged_out, (__half*)st->ofmap, st->perm, (const __half*)bias, num_pos, st->F));
    }
    CK(cudaGetLastError());
    return SHFLBW_OK;
}

int shflbw_spconv_launches_per_exec(const shflbw_spconv_state_t* st) {
    if (!st || !st->init_success) return 0;
    if (st->kernel == SHFLBW_KERNEL_SIMT || st->chain) return 1;
    return st->staged_out ? 3 : 2;
}

// Host-buffer SpConv.  Batches of 32 images or more go in up to four chunks of whole 8-image
// groups (NHWC: a batch slice is contiguous on both sides) through the same three streams as
// the SpMM host call, so that copy in, kernels and copy out overlap.
int shflbw_spconv_host(shflbw_matrix_t* f, int B, int Hin, int Win, int stride, const void* ifmap_host,
                       void* ofmap_host, float alpha) {
    if (!f || !ifmap_host || !ofmap_host || !f->is_filter || B <= 0 || Hin <= 0 || Win <= 0 || stride <= 0)
        return SHFLBW_ERR_INVALID_ARG;
    int rc = shflbw_matrix_to_device(f);
    if (rc != SHFLBW_OK) return rc;
    if (!on_current_device(*f)) return SHFLBW_ERR_NOT_ON_DEVICE;   // before staging buffers / streams are made
    const int Ho = (Hin + stride - 1) / stride, Wo = (Win + stride - 1) / stride;
    const size_t img_in = (size_t)Hin * Win * f->C, img_out = (size_t)Ho * Wo * f->F;   // elements per image
    if ((rc = ensure_buffer(&f->stage_in, &f->stage_in_bytes, (size_t)B * img_in * 2)) != SHFLBW_OK) return rc;
    if ((rc = ensure_buffer(&f->stage_out, &f->stage_out_bytes, (size_t)B * img_out * 2)) != SHFLBW_OK) return rc;
    int per = B;                                     // images per chunk
    if (B >= 32) per = ((B + 3) / 4 + 7) / 8 * 8;
    const int chunks = (B + per - 1) / per;          // <= 4
    cudaStream_t s_in, s_k, s_out;
    cudaEvent_t *e_in, *e_k;
    if ((rc = host_pipeline(f, &s_in, &s_k, &s_out, &e_in, &e_k)) != SHFLBW_OK) return rc;
    auto fail = [&](int code) { cudaDeviceSynchronize(); return code; };
#define CKH(call) do { if (!cuda_ok((call), #call)) return fail(SHFLBW_ERR_CUDA); } while (0)
    for (int i = 0; i < chunks; ++i) {
        const int b0 = i * per, nb = (B - b0 < per) ? B - b0 : per;
        __half* dI = (__half*)f->stage_in + (size_t)b0 * img_in;
        __half* dO = (__half*)f->stage_out + (size_t)b0 * img_out;
        CKH(cudaMemcpyAsync(dI, (const __half*)ifmap_host + (size_t)b0 * img_in, (size_t)nb * img_in * 2,
                            cudaMemcpyHostToDevice, s_in));
        CKH(cudaEventRecord(e_in[i], s_in));
        CKH(cudaStreamWaitEvent(s_k, e_in[i], 0));
        shflbw_spconv_state_t st;
        rc = shflbw_spconv_init(f, nb, Hin, Win, stride, dI, dO, alpha, SHFLBW_KERNEL_AUTO, &st);
        if (rc == SHFLBW_OK) rc = shflbw_spconv_exec(&st, s_k);
        if (rc != SHFLBW_OK) return fail(rc);
        CKH(cudaEventRecord(e_k[i], s_k));
        CKH(cudaStreamWaitEvent(s_out, e_k[i], 0));
        CKH(cudaMemcpyAsync((__half*)ofmap_host + (size_t)b0 * img_out, dO, (size_t)nb * img_out * 2,
                            cudaMemcpyDeviceToHost, s_out));
    }
    CKH(cudaStreamSynchronize(s_out));
    CKH(cudaStreamSynchronize(s_k));
    CKH(cudaStreamSynchronize(s_in));
#undef CKH
    return SHFLBW_OK;
}

// ---- chained layers ---------------------------------------------------------------------

size_t shflbw_chain_buffer_elems(int C, int H, int W, int B, int R, int S) {
    if (C <= 0 || H <= 0 || W <= 0 || B <= 0 || R <= 0 || S <= 0) return 0;
    return (size_t)C * (H + R - 1) * (W + S - 1) * ((B + 7) / 8 * 8);
}

int shflbw_chain_import_nhwc(const void* nhwc, int B, int H, int W, int C, int R, int S, void* chain_buf,
                             void* stream) {
    if (!nhwc || !chain_buf || B <= 0 || H <= 0 || W <= 0 || C <= 0 || R <= 0 || S <= 0) return SHFLBW_ERR_INVALID_ARG;
    if (C % 8 || (((uintptr_t)nhwc | (uintptr_t)chain_buf) & 15)) return SHFLBW_ERR_UNSUPPORTED;
    if ((long long)shflbw_chain_buffer_elems(C, H, W, B, R, S) >= (1ll << 31)) return SHFLBW_ERR_UNSUPPORTED;
    launch_relayout((const __half*)nhwc, (__half*)chain_buf, B, (B + 7) / 8 * 8, H, W, C, R, S, (cudaStream_t)stream);
    CK(cudaGetLastError());
    return SHFLBW_OK;
}

int shflbw_chain_export_nhwc(const void* chain_buf, int B, int H, int W, int F, int R, int S,
                             const shflbw_matrix_t* producer, void* nhwc, void* stream) {
    if (!chain_buf || !nhwc || B <= 0 || H <= 0 || W <= 0 || F <= 0 || R <= 0 || S <= 0) return SHFLBW_ERR_INVALID_ARG;
    if (F % 8 || (((uintptr_t)nhwc | (uintptr_t)chain_buf) & 15)) return SHFLBW_ERR_UNSUPPORTED;
    const int* perm = nullptr;
    if (producer) {
        if (producer->nrow != F) return SHFLBW_ERR_BAD_FORMAT;
        if (!on_current_device(*producer)) return SHFLBW_ERR_NOT_ON_DEVICE;
        perm = producer->d_perm;
    }
    if (F > 14528) return SHFLBW_ERR_UNSUPPORTED;           // the documented range; the kernel itself needs grid.y = F / 64 <= 65535
    const int Bp = (B + 7) / 8 * 8;
    if ((long long)H * W * (Bp / 8) >= (1ll << 31)) return SHFLBW_ERR_UNSUPPORTED;
    CK(launch_export(chain_buf, nhwc, perm, B, Bp, H, W, H + R - 1, W + S - 1, R / 2, S / 2, F, (cudaStream_t)stream));
    CK(cudaGetLastError());
    return SHFLBW_OK;
}

int shflbw_spconv_chain_init(shflbw_matrix_t* f, int B, int Hin, int Win, int stride, const void* in_chain,
                             void* out_chain, int R_next, int S_next, float alpha, int relu,
                             shflbw_spconv_state_t* out) {
    if (!out) return SHFLBW_ERR_INVALID_ARG;
    std::memset(out, 0, sizeof *out);
    if (!f || !in_chain || !out_chain || B <= 0 || Hin <= 0 || Win <= 0 || stride <= 0 || R_next <= 0 || S_next <= 0)
        return SHFLBW_ERR_INVALID_ARG;
    if (!f->is_filter) return SHFLBW_ERR_INVALID_ARG;
    if (!on_current_device(*f)) return SHFLBW_ERR_NOT_ON_DEVICE;
    if (f->brow != 32 && f->brow != 64 && f->brow != 128) return SHFLBW_ERR_UNSUPPORTED;
    if (f->C % 8 || !f->d_kcrs) return SHFLBW_ERR_UNSUPPORTED;
    if (((uintptr_t)in_chain | (uintptr_t)out_chain) & 15) return SHFLBW_ERR_UNSUPPORTED;
    const int Ho = (Hin + stride - 1) / stride, Wo = (Win + stride - 1) / stride;
    const int Bp = (B + 7) / 8 * 8;
    const long long tokens = (long long)Ho * Wo * Bp;
    // 32-bit element offsets into both chain buffers
    if (tokens >= (1ll << 31) || (long long)shflbw_chain_buffer_elems(f->C, Hin, Win, B, f->R, f->S) >= (1ll << 31) ||
        (long long)shflbw_chain_buffer_elems(f->F, Ho, Wo, B, R_next, S_next) >= (1ll << 32) - 1)
        return SHFLBW_ERR_UNSUPPORTED;
    out->B = B; out->Hin = Hin; out->Win = Win; out->C = f->C; out->F = f->F; out->R = f->R; out->S = f->S;
    out->stride = stride; out->Ho = Ho; out->Wo = Wo; out->V = f->brow; out->Bp = Bp;
    out->alpha = alpha; out->ifmap = in_chain; out->ofmap = out_chain;
    out->blk_ptr = f->d_kptr; out->blk_idx = f->d_kcrs; out->blk_val = f->d_val;
    out->perm = f->d_perm; out->status_word = f->d_status;
    out->chain = 1; out->out_R = R_next; out->out_S = S_next; out->relu = relu != 0;
    PanelChoice ch;
    const int row_blocks = f->F / f->brow;
    const long long padded_cols = f->kptr.empty() ? 0 : f->kptr.back();
    const ConvTokens ct = conv_tokens(Ho, Wo, Win + f->S - 1, Bp, stride, f->brow, row_blocks, padded_cols, true);
    const long long counted = (long long)Ho * ct.row_pix * Bp;
    const int tile = pick_tile(counted, row_blocks);
    const long long items = (counted + tile - 1) / tile * row_blocks;
    const bool rows = chain_rows(f->brow, S_next > 1 && tma_row_pix(Wo, Win + f->S - 1, Bp, stride) > Wo, items, padded_cols, row_blocks);
    const int ring = !rows && chain_wide(f->brow, tile, items, padded_cols, row_blocks) ? wide_ring_of(false, padded_cols, row_blocks) : 0;
    int rc = pick_panel<shflbw::kPanelConvChain>(f->brow, tile, rows, ring, ct.gather, &ch);
    if (rc != SHFLBW_OK) return rc;
    out->kernel = SHFLBW_KERNEL_TCGEN05;
    out->tokens_per_cta = ch.tokens; out->stages = ch.stages; out->producer_warps = ch.pw; out->variant = ch.variant;
    out->gather = ch.gather; out->row_pix = ct.row_pix; out->rows = rows; out->wide = ch.variant == 2;
    out->tiles_n = (int)((counted + ch.tokens - 1) / ch.tokens);
    out->num_items = out->tiles_n * row_blocks;
    const int sms = sm_count();
    if (sms <= 0) return SHFLBW_ERR_CUDA;
    out->block_x = ch.threads;
    out->grid_x = persistent_grid(out->num_items, sms); out->grid_y = 1;
    out->shared_mem_size = ch.smem;
    out->init_success = 1;
    return SHFLBW_OK;
}

int shflbw_chain_residual_map(const shflbw_matrix_t* layer, const shflbw_matrix_t* producer, int* map_host) {
    if (!layer || !map_host) return SHFLBW_ERR_INVALID_ARG;
    const int F = layer->nrow;
    if (producer && producer->nrow != F) return SHFLBW_ERR_BAD_FORMAT;
    std::vector<int> where(F);      // logical channel -> plane of the residual buffer
    for (int p = 0; p < F; ++p) where[producer && producer->row_permute ? producer->row_permute_ids[p] : p] = p;
    for (int f = 0; f < F; ++f) map_host[f] = where[layer->row_permute ? layer->row_permute_ids[f] : f];
    return SHFLBW_OK;
}

int shflbw_spconv_chain_set_residual(shflbw_matrix_t* f, shflbw_spconv_state_t* st, const void* res_chain,
                                     const int* map_host) {
    if (!f || !st || !st->init_success || !st->chain || !res_chain) return SHFLBW_ERR_INVALID_ARG;
    if (!on_current_device(*f) || st->blk_ptr != f->d_kptr) return SHFLBW_ERR_INVALID_ARG;
    if ((uintptr_t)res_chain & 15) return SHFLBW_ERR_UNSUPPORTED;
    if (map_host)
        for (int i = 0; i < st->F; ++i)
            if (map_host[i] < 0 || map_host[i] >= st->F) return SHFLBW_ERR_BAD_FORMAT;
    // The sixteen-epilogue-warp kernel copies the residual an item ahead, which pays up to two stages of
    // columns per block (14x14x256 -> 1024 with residual, batch 128, 112 columns: 33.9 -> 26.5 us); without a
    // residual the limit is one stage (pick_panel).  Where the residual's rows come in whole boxes the copy engine
    // fetches them (by cp.async and by TMA, 51 columns a block or fewer, back to back: 56x56x64 -> 256, batch 256 183 and
    // 158 us, 118 73.1 and 70.0, 64 40.7 and 39.2; 14x14x256 -> 1024, batch 256 47.7 and 41.3, 118 23.8 and 21.4;
    // 28x28x128 -> 512, batch 256 87.5 and 84.0 in the network, 84.0 and 87.1 alone, 118 39.3 and 36.9; 7x7x512 -> 2048, 256
    // 27.3 and 26.4; a network of batch 256 2427 and 2298, 64 759 and 745, 32 501 and 499), with three gather warps, from six items
    // per SM on; with fewer the slots' first laps are most of it (5.3 items per SM, 56x56x64 -> 256, batch 16: 12.1 and
    // 12.5; 2.7, 28x28x128 -> 1024, batch 8, 60 columns: eight warps 9.38, sixteen by cp.async 9.02, by TMA 9.64).
    PanelChoice ch;
    const long long padded_cols = f->kptr.empty() ? 0 : f->kptr.back();
    const bool two_warps = padded_cols <= 48ll * (st->F / st->V) && (long long)st->F * st->Ho * st->Wo * st->Bp * 2 <= (256ll << 20);   // (lookup)
    const int eb = tuned("SHFLBW_BOX");                      // 0: residual by cp.async (tuning aid)
    const bool box = st->gather == shflbw::kGatherTma && boxes_fit(*st) && (eb != kUnset ? eb != 0 : st->num_items >= 6ll * sm_count());
    const bool wide = (st->variant == 2 ||
                       (st->variant == 0 && st->V == 64 && st->tokens_per_cta == 256 && tuned("SHFLBW_EPILOGUE_WARPS") == kUnset &&
                        padded_cols <= 128ll * (st->F / st->V) && 2ll * st->num_items >= 5ll * sm_count())) &&
                      lookup<shflbw::kPanelConvChain>(64, 256, &ch, st->gather, 6, two_warps ? 2 : 3, box);
    if (wide) {
        const int rc = allow_smem(ch.fn, ch.smem);
        if (rc != SHFLBW_OK) return rc;
    }
    const int* map_dev = nullptr;
    if (map_host) {
        // One device buffer per state: re-binding the residual of the same state (every step,
        // say) overwrites the map of an earlier call, one of the handle's retired buffers, in place
        // instead of allocating again.
        void* d = nullptr;
        for (void* r : f->retired) if (r == (const void*)st->residual_map) d = r;
        if (!d) {
            CK(cudaMalloc(&d, (size_t)st->F * sizeof(int)));
            f->retired.push_back(d);                   // lives as long as the filter's device copy
        }
        CK(cudaMemcpy(d, map_host, (size_t)st->F * sizeof(int), cudaMemcpyHostToDevice));
        map_dev = (const int*)d;
    }
    // Nothing can fail from here on: a refused call leaves the state as it was.
    st->residual = res_chain;
    st->residual_map = map_dev;
    st->box_res = wide && box;
    if (wide) {
        st->variant = 2; st->wide = 1; st->stages = ch.stages; st->producer_warps = ch.pw; st->block_x = ch.threads; st->shared_mem_size = ch.smem;
    }
    return SHFLBW_OK;
}

int shflbw_spconv_exec_static_scratch(const shflbw_matrix_t* f, int B, int Hin, int Win, int stride,
                                      const void* ifmap, void* ofmap, float alpha, void* stream) {
    // Same argument checks, 32-bit range checks and launch plan as shflbw_spconv_init (with an
    // unpermuted filter the output can bypass the array, so its capacity alone would not bound
    // the output offsets); only the scratch comes from somewhere else.
    shflbw_spconv_state_t st;
    int rc = plan_conv(f, B, Hin, Win, stride, ifmap, ofmap, alpha, SHFLBW_KERNEL_TCGEN05, &st, SHFLBW_STATIC_SCRATCH_BYTES);
    if (rc != SHFLBW_OK) return rc;

    // Capacity check first: nothing is launched when the shape does not fit.
    auto up256 = [](unsigned long long v) { return (v + 255ull) / 256ull * 256ull; };
    const unsigned long long in_bytes = up256(st.staged_in_bytes), out_bytes = up256(st.staged_out_bytes);
    if (in_bytes + out_bytes > (unsigned long long)SHFLBW_STATIC_SCRATCH_BYTES) {
        snprintf(g_cuda_err, sizeof g_cuda_err,
                 "static scratch: this shape needs %llu bytes, the built-in array holds %u",
                 in_bytes + out_bytes, (unsigned)SHFLBW_STATIC_SCRATCH_BYTES);
        return SHFLBW_ERR_TOO_LARGE;
    }

    // Once per device, with that device current: the array's device address.
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return SHFLBW_ERR_UNSUPPORTED;
    if (!g_static_scratch_addr[dev]) {
        void* ptr = nullptr;
        CK(cudaGetSymbolAddress(&ptr, g_static_scratch));
        if (!ptr) return SHFLBW_ERR_CUDA;
        g_static_scratch_addr[dev] = ptr;
    }
    unsigned char* scratch = (unsigned char*)g_static_scratch_addr[dev];
    st.staged_in = scratch;
    if (st.staged_out_bytes) st.staged_out = scratch + in_bytes;
    st.init_success = 1;
    return shflbw_spconv_exec(&st, stream);
}

// ---- several GPUs from one process -------------------------------------------------------

struct shflbw_multi {
    struct Shard {
        int device = -1;
        shflbw_matrix_t* mat = nullptr;      // replica of the sparse operand on `device`
        cudaStream_t stream = nullptr;
        cudaEvent_t start = nullptr, stop = nullptr;
        int kind = 0;                        // 0 none, 1 SpMM, 2 SpConv
        shflbw_spmm_state_t spmm;
        shflbw_spconv_state_t conv;
    };
    std::vector<Shard> shards;
};

namespace {
struct DeviceGuard {                         // restores the caller's current device
    int prev = -1;
    DeviceGuard() { cudaGetDevice(&prev); }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};
}  // namespace

int shflbw_multi_create(const shflbw_matrix_t* m, const int* device_ids, int n, shflbw_multi_t** out) {
    if (!m || !device_ids || n <= 0 || n > kMaxDevices || !out) return SHFLBW_ERR_INVALID_ARG;
    *out = nullptr;
    int have = 0;
    CK(cudaGetDeviceCount(&have));
    for (int g = 0; g < n; ++g) if (device_ids[g] < 0 || device_ids[g] >= have) return SHFLBW_ERR_INVALID_ARG;
    DeviceGuard guard;
    auto* mg = new shflbw_multi;
    mg->shards.resize(n);
    int rc = SHFLBW_OK;
    for (int g = 0; g < n && rc == SHFLBW_OK; ++g) {
        auto& sh = mg->shards[g];
        sh.device = device_ids[g];
        if (!cuda_ok(cudaSetDevice(sh.device), "cudaSetDevice")) { rc = SHFLBW_ERR_CUDA; break; }
        if ((rc = shflbw_matrix_clone(m, &sh.mat)) != SHFLBW_OK) break;
        if ((rc = shflbw_matrix_to_device(sh.mat)) != SHFLBW_OK) break;
        if (!cuda_ok(cudaStreamCreateWithFlags(&sh.stream, cudaStreamNonBlocking), "cudaStreamCreate") ||
            !cuda_ok(cudaEventCreate(&sh.start), "cudaEventCreate") || !cuda_ok(cudaEventCreate(&sh.stop), "cudaEventCreate"))
            rc = SHFLBW_ERR_CUDA;
    }
    if (rc != SHFLBW_OK) { shflbw_multi_destroy(mg); return rc; }
    *out = mg;
    return SHFLBW_OK;
}

void shflbw_multi_destroy(shflbw_multi_t* mg) {
    if (!mg) return;
    DeviceGuard guard;
    for (auto& sh : mg->shards) {
        if (sh.device >= 0) cudaSetDevice(sh.device);
        if (sh.stream) { cudaStreamSynchronize(sh.stream); cudaStreamDestroy(sh.stream); }
        if (sh.start) cudaEventDestroy(sh.start);
        if (sh.stop) cudaEventDestroy(sh.stop);
        shflbw_matrix_destroy(sh.mat);
    }
    delete mg;
}

int shflbw_multi_shards(const shflbw_multi_t* mg) { return mg ? (int)mg->shards.size() : 0; }

int shflbw_multi_spmm_init(shflbw_multi_t* mg, const int* n_per_shard, const void* const* B, void* const* D, float alpha) {
    if (!mg || !n_per_shard || !B || !D) return SHFLBW_ERR_INVALID_ARG;
    DeviceGuard guard;
    for (size_t g = 0; g < mg->shards.size(); ++g) {
        auto& sh = mg->shards[g];
        sh.kind = 0;
        if (n_per_shard[g] == 0) continue;                    // an empty shard is legal: nothing to launch
        CK(cudaSetDevice(sh.device));
        const int rc = shflbw_spmm_init(sh.mat, n_per_shard[g], B[g], alpha, nullptr, 0.f, D[g], SHFLBW_KERNEL_AUTO, &sh.spmm);
        if (rc != SHFLBW_OK) return rc;
        sh.kind = 1;
    }
    return SHFLBW_OK;
}

int shflbw_multi_spconv_init(shflbw_multi_t* mg, const int* images_per_shard, int Hin, int Win, int stride,
                             const void* const* ifmap, void* const* ofmap, float alpha) {
    if (!mg || !images_per_shard || !ifmap || !ofmap) return SHFLBW_ERR_INVALID_ARG;
    DeviceGuard guard;
    for (size_t g = 0; g < mg->shards.size(); ++g) {
        auto& sh = mg->shards[g];
        sh.kind = 0;
        if (images_per_shard[g] == 0) continue;
        CK(cudaSetDevice(sh.device));
        const int rc = shflbw_spconv_init(sh.mat, images_per_shard[g], Hin, Win, stride, ifmap[g], ofmap[g], alpha,
                                          SHFLBW_KERNEL_AUTO, &sh.conv);
        if (rc != SHFLBW_OK) return rc;
        sh.kind = 2;
    }
    return SHFLBW_OK;
}

int shflbw_multi_exec(shflbw_multi_t* mg) {
    if (!mg) return SHFLBW_ERR_INVALID_ARG;
    DeviceGuard guard;
    for (auto& sh : mg->shards) {                              // back to back: nothing here waits for a GPU
        if (!sh.kind) continue;
        CK(cudaSetDevice(sh.device));
        CK(cudaEventRecord(sh.start, sh.stream));
        const int rc = sh.kind == 1 ? shflbw_spmm_exec(&sh.spmm, sh.stream) : shflbw_spconv_exec(&sh.conv, sh.stream);
        if (rc != SHFLBW_OK) return rc;
        CK(cudaEventRecord(sh.stop, sh.stream));
    }
    return SHFLBW_OK;
}

int shflbw_multi_sync(shflbw_multi_t* mg, float* max_ms) {
    if (!mg) return SHFLBW_ERR_INVALID_ARG;
    DeviceGuard guard;
    float worst = 0.f;
    int status = SHFLBW_OK;
    for (auto& sh : mg->shards) {
        CK(cudaSetDevice(sh.device));
        CK(cudaStreamSynchronize(sh.stream));
        if (sh.kind) {
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, sh.start, sh.stop) == cudaSuccess && ms > worst) worst = ms;
            else (void)cudaGetLastError();
            const int rc = shflbw_matrix_device_status(sh.mat);
            if (rc != SHFLBW_OK) status = rc;
        }
    }
    if (max_ms) *max_ms = worst;
    return status;
}

}  // extern "C"
