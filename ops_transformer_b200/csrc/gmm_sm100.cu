// Grouped int8 GEMM for sm_100a: TMA-staged tiles -> tcgen05.mma kind::i8 -> TMEM int32 accumulators ->
// warp-specialised fused epilogue.  Persistent CTA pairs (one CTA per SM) walk a tile list that every CTA derives
// from group_list on the device (empty experts produce no tiles).
//
// Replaces, for NVIDIA B200, the reference's AscendC kernels
//   gmm/grouped_matmul/op_kernel/grouped_matmul.h:250-283            (GMMProcess::Process, the block scheduler)
//   gmm/grouped_matmul/op_kernel/grouped_matmul_quant_mixcore.h:175-315 (int8 matmul + dequant epilogue)
//   gmm/grouped_matmul_swiglu_quant/op_kernel/grouped_matmul_swiglu_quant.h:231-262, 367-474 (matmul, dequant, SwiGLU)
// and the host tiling that feeds them (op_host/op_tiling/grouped_matmul_tiling.cpp:727-763).
//
// Orientation: the weight columns ("channels") are the M side of the MMA, 128 per CTA (a TMEM lane is a channel); the
// token rows are its N side, any multiple of 32 up to 256 (a TMEM column is a token).  A group of R rows is cut into
// ceil(R / 256) tiles of nearly equal size, so what a tile costs follows the rows it has: with the tokens on the M side
// a group's last tile multiplied up to 255 rows of other groups (12.5 % of all MMA work on 32 groups of ~1024 rows, half
// of it on groups of ~250), and a decode tile of a few rows staged and multiplied 128.
//   grouped_matmul       : a CTA's 128 channels are 128 consecutive output columns.
//   swiglu_quant, pairs  : lanes [0,64) are weight columns j0.. (activated half), lanes [64,128) are N/2+j0.. (linear
//                          half): a tile yields 64 outputs per CTA and token; the two halves meet through shared memory.
//   swiglu_quant, one CTA: both halves of 128 columns in two accumulators of at most 128 tokens; a lane holds both values.
// K is consumed 128 bytes per pipeline stage (4 MMAs of K=32).
// Warp roles: warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer, warps 2-9 = epilogue (320 threads; with bias or
// activation warps 2-17, 576 threads); swiglu_quant adds warp 10, one lane of which keeps the books of the row blocks in global
// memory, and requantising warps up to 512 threads; FRACTAL_NZ adds two weight loader warps (in swiglu_quant they take the
// place of two requantising warps).
// CTA pairs (cluster of 2, tcgen05 cta_group::2) compute 256 channels; each CTA stages its own 128 channels and half of the
// tile's token rows.  A launch confined to one CTA runs the one-CTA instances.  Weight layouts: [E,K,N] (MN-major operand,
// 128-byte swizzle; 64-byte for swiglu's 64-channel boxes), the transposed view [E,N,K] (K-major) and FRACTAL_NZ
// [E,N/32,K/16,16,32] (MN-major, 32-byte swizzle, fetched by two loader warps instead of TMA).
// Epilogue: a lane holds one channel (its weight scale stays in a register), the tokens' scales come from shared memory.
// bf16 / fp16 results are read as 16x256b fragments, packed by token pairs and transposed by stmatrix, so that the four
// warps of a column half together hold 256 contiguous bytes of every result row; SwiGLU values are stored as they are held, a
// token's 32 channels (128 bytes) per instruction; the combine's fp32 rows and int32 accumulators are transposed 16 tokens at
// a time, so that a lane adds or stores four channels of a row at once.
// Rows are optionally scattered by a row index, also into other GPUs' buffers; the finalize-routing variant adds weighted
// fp32 rows into token rows with 16-byte vector reductions; SwiGLU values go to an fp32 staging buffer with a per-row
// atomic max, and a finished row block is requantised to int8 in row slices that the CTAs which worked on it claim from a
// counter - no CTA ever waits for another one (see publish_and_collect).
// What bounds it: long groups the power limit (the MMA loop runs at 550-570 cycles per K block of 512 where the epilogue is
// idle; the SM clock falls to 1.5-1.6 GHz, at which the tensor pipe alone draws the board's 1 kW); groups of up to 128 rows
// HBM; short K the epilogue.  Measured before (tokens on the M side, operations issued by one thread of a diverged warp,
// every epilogue thread fencing for itself, requantisation inside the epilogue warps) and now, us:
//   swiglu K=7168 N=4096: 4096 tokens x 8 over 32 experts 892 / 886 (power), 128 tokens x 8 over 256 experts 884 / 850 (HBM);
//     K=2048 N=1536, 64 groups of 64 rows 66 / 52, of 400 rows 190 / 112
//   gmm K=2048 N=7168: 4096 tokens x 8 over 32 experts 403 / 366; 32 groups of 160 rows 131 / 96; K=768 N=2048, 64 x 400 rows
//     76 / 60 (of which 10 % came from moving the second CTA's accumulator release out of its epilogue warps: 374 / 334 for
//     32 groups of 1000 rows)
// The producers pace themselves wave by wave so that the units which share x rows and weight boxes through L2 stay
// together (a bounded hint).
// Every wait on an mbarrier is bounded; on expiry the CTA records a status word, all roles leave their loops,
// outstanding copies are drained with a second bounded wait, TMEM is released and the kernel returns.
// -DGMM_TRACE builds in clock64 / globaltimer stamps of the roles of a few CTAs (a buffer address comes from the environment).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstddef>
#include <cstdlib>

#include "gmm_common.h"

namespace gmm {
namespace {

constexpr int BC = 128;                 // channels (weight columns) per CTA: the MMA's M side, one TMEM lane each
constexpr int BT = 256;                 // most tokens of a tile: the MMA's N side, one TMEM column each
constexpr int TOK_STEP = 32;            // the MMA's N is a multiple of this
constexpr int SPLIT_TOK = 64;           // the last wave's tiles are cut no further than brings the largest tile to this
constexpr int BK = 128;
constexpr int UMMA_K = 32;
constexpr int W_STAGE = BC * BK;        // a CTA's channels x 128 bytes of K
constexpr int PIPE_BYTES = 196608;      // shared memory given to the TMA ring
constexpr int MAX_STAGES = 6;
constexpr int X_MAPS = 3;               // tensor maps of x with boxes of 32, 64 and 128 rows

// CTAS = 2: a pair of CTAs (one cluster) computes 256 channels with cta_group::2 MMAs; each CTA stages its own 128 channels
//           (16 KB per K block) and half of the tile's tokens (at most 16 KB).  The pair's even CTA issues the MMAs for both.
// CTAS = 1: one CTA, 128 channels, all tokens of the tile (at most 32 KB).
//   swiglu_quant: 128 channels of either half (32 KB) into two accumulators of at most 128 tokens each, so that a lane holds
//   both values of its column.
// The ring has as many stages as PIPE_BYTES holds of the launch's largest token box, at most MAX_STAGES.
template <int MODE, int CTAS>
struct Shape {
    static constexpr bool kDual = MODE == kModeSwigluQuant && CTAS == 1;
    static constexpr int kWStage = kDual ? 2 * W_STAGE : W_STAGE;
    static constexpr int kMaxTok = kDual ? BT / 2 : BT;
    static constexpr int kCols = MODE == kModeSwigluQuant && !kDual ? BC / 2 : BC;   // result columns per CTA and tile
};
// Row blocks of a group that are worked on together: all their tiles of a channel tile, then the next channel tile.  A group that
// begins in one wave and ends in the next has its x rows read twice then, instead of its weights, four times as many (DRAM reads
// of 8 groups of 1024 rows, K=7168 N=4096: 403 -> 330 MB).  It is traffic that this saves: the kernel's time stays within the
// runs' spread, also where four blocks have more tiles than a wave has units (swiglu, us with one / two / four: K=7168 N=4096, 32
// groups of 1024 rows 664 / 672 / 662; K=4096 N=8192, 16 of 2048 rows 806 / 801 / 796; K=4096 N=10240, 4 of 1024 rows 204 / 191 /
// 196).  grouped_matmul, which does not pace its waves, K=2048 N=7168: 339 / - / 343.
__host__ __device__ constexpr int block_group(int mode) { return mode == kModeSwigluQuant ? 4 : 1; }
constexpr int MAX_GROUPS = 1024;
enum : int { kEpiPlain = 0, kEpiScatter = 1, kEpiGeneric = 2, kEpiCombine = 3, kEpiHalf = 4, kEpiHalfScatter = 5 };
// Epilogue warps, and the tokens of the chunks that they take in turns: two warps per TMEM lane quarter and 32 tokens; with
// options (bias, activation) four and 16.  The options' chains of dependent instructions left the schedulers idle with two warps
// each (K=1424 N=2976, 3055 rows, fp16, bias, GELU: 38.8 us, now 37.4; K=2048 N=2048, 16 groups of 250 rows, bias, SiLU: 36.7 /
// 35.2); the plain epilogue, which the MMAs hide, only got in their way (K=2048 N=7168, 32 groups of 1024 rows: 360 / 364).
__host__ __device__ constexpr bool wide_epilogue(int mode, int epi) { return mode == kModeDequantBf16 && epi == kEpiGeneric; }
__host__ __device__ constexpr int epi_warps(int mode, int epi) { return wide_epilogue(mode, epi) ? 16 : 8; }
__host__ __device__ constexpr int chunk_tokens(int mode, int epi) { return wide_epilogue(mode, epi) ? 16 : 32; }
// swiglu_quant only: one more warp, of which one lane keeps the books of the row blocks in global memory (arrivals, slice
// claims) beside the epilogue, so that none of its round trips to L2 delays the next tile.  It hands the requantising warps
// lists of row ranges through a small ring.
constexpr int WK_DEPTH = 4;                  // work lists the publishing lane may be ahead of the requantising warps
// Weight loader warps (FRACTAL_NZ only).  A 32-byte row of that storage is a row of its own to TMA, 512 per 16 KB, and the
// copy engine takes about 1.75 cycles for each: 900 cycles per K block where the MMAs need 512 and HBM 740.  In memory 128
// K-rows of a 32-column slab are 4 KB in one piece, so two warps fetch them with 16-byte cp.async, 512 contiguous bytes per
// instruction, and put the halves of every row where the 32-byte swizzle wants them.  Tensor copies / loader warps, us:
// K=2048 N=7168 with 128 tokens x 8 over 256 experts 532 / 418 (6.6 TB/s), swiglu K=7168 N=4096 with 4096 tokens x 8 over 32
// experts 955 / 844, gmm K=2048 N=7168 with 32 x 400 rows 204 / 184.
constexpr int LD_WARPS = 2;
__host__ __device__ constexpr int ld_warps(int bl) { return bl == 2 /* kBFractalNz */ ? LD_WARPS : 0; }
// swiglu_quant: warps that requantise finished row blocks beside the epilogue; with 16 warps in all a thread has 128 registers
__host__ __device__ constexpr int rq_warps(int bl) { return 5 - ld_warps(bl); }
__host__ __device__ constexpr int num_threads(int mode, int bl, int epi)
{
    return 64 + 32 * epi_warps(mode, epi) + 32 * ld_warps(bl) + (mode == kModeSwigluQuant ? 32 + 32 * rq_warps(bl) : 0);
}
constexpr int TMEM_COLS = 512;
constexpr long long WAIT_LIMIT_CYCLES = 1ll << 31;   // about a second
constexpr long long DRAIN_LIMIT_CYCLES = 1ll << 24;  // a few milliseconds
// Upper bound (ns) of the time a thread may stay suspended inside one mbarrier.try_wait before it polls again.  The board
// is power capped under these kernels, so waiting warps that poll less leave more of the budget to the clock: with 2 us
// instead of the default C3 runs 0.399 instead of 0.414 ms, C2 0.80-0.81 instead of 0.82-0.83 ms (same box, alternating).
constexpr uint32_t WAIT_SUSPEND_NS = 2000;

// Weight layouts: [E,K,N]; [E,N,K] (the transposed view); FRACTAL_NZ [E, N/32, K/16, 16, 32] (32-byte runs along N).
enum : int { kBRowMajor = 0, kBTransposed = 1, kBFractalNz = 2 };
constexpr int MAX_PENDING = 6;         // unsettled row blocks a CTA keeps track of before it hands its share over
// Epilogue staging: 32-bit results 16 tokens x 128 bytes per warp; 16-bit results 64 tokens of 256 bytes each (a chunk for
// every four warps), 16 bytes apart so that the eight 16-byte rows of a stmatrix fall into different banks.
constexpr int WARP_STAGE_BYTES = 2048;
constexpr int ROW16_PITCH = 2 * BC + 16;
constexpr int OUT_STAGE_BYTES = 64 * ROW16_PITCH;
static_assert(OUT_STAGE_BYTES >= 8 * WARP_STAGE_BYTES, "one staging area serves both forms");

// A row block some of whose S this CTA has stored (swiglu_quant).
struct PendingBlock {
    int rb, row0, rows;
    int weight, shares;                // the CTA's shares of the block's requantisation, and how many there are
};

struct Shared {
    uint64_t full[MAX_STAGES];
    uint64_t empty[MAX_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t tok_ready[2];             // all epilogue threads have stored their token's scale
    uint64_t grp_sync[4];              // epilogue warps that exchange values through out_stage (see group_sync)
    uint64_t wk_full[WK_DEPTH];        // a work list is written (swiglu_quant)
    uint64_t wk_empty[WK_DEPTH];       // every requantising warp is done with it
    int closing_slot;                  // the ring slot of the last list
    uint64_t wk_closing;               // the last list is written (for the epilogue warps, which help with that one)
    uint32_t tmem_base;
    int abort_flag;
    int total_tiles;
    int max_tok;                       // tokens of the largest tile
    int split_from, split;             // tiles from split_from on are cut into `split` pieces of their tokens (see build_schedule)
    long long wait_limit;              // bound of every wait, in cycles
    // swiglu_quant: how many epilogue warps have stored their part of how many tiles; the row blocks this
    // CTA contributed to and has not yet settled (publishing lane only); a ring of work lists: the row ranges to requantise
    // (written by that lane, read by the requantising warps after wk_full)
    unsigned stored_count;
    unsigned published;                // tiles that the publishing lane is done with (see list_wait)
    int pend_n;
    PendingBlock pend[MAX_PENDING];
    int n_work[WK_DEPTH];
    int work_last[WK_DEPTH];           // no list follows
    int work_begin[WK_DEPTH][MAX_PENDING + 1], work_end[WK_DEPTH][MAX_PENDING + 1];
    int row_start[MAX_GROUPS];
    int rows[MAX_GROUPS];
    int tile_start[MAX_GROUPS + 1];
    // per accumulator buffer: the factor of every token of the tile (x scale, for the combine times the routing weight) and
    // the combine's routing weight on its own (for the bias term).  A buffer is written after acc_full of its tile, i.e.
    // after every epilogue warp has left the tile before last, which used it.
    alignas(16) float tok_scale[2][BT];
    alignas(16) float tok_logit[2][BT];
    alignas(16) uint8_t out_stage[OUT_STAGE_BYTES];
};

constexpr size_t SMEM_BYTES = 1024 + (size_t)PIPE_BYTES + sizeof(Shared);
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
static_assert(offsetof(Shared, tok_scale) % 16 == 0 && offsetof(Shared, out_stage) % 16 == 0, "vector accesses need 16-byte alignment");

// Debug build only (-DGMM_TRACE): clock64 stamps of the roles of a few CTAs, written to a buffer whose address comes from
// the environment; layout [cta < 4][role < 4][tile < 64][slot < 8].
#ifdef GMM_TRACE
#define TRACE(role, tile, slot)                                                                                           \
    do {                                                                                                                  \
        if (p.trace && blockIdx.x < 4 && (tile) < 64) p.trace[(((int)blockIdx.x * 4 + (role)) * 64 + (tile)) * 8 + (slot)] = clock64(); \
    } while (0)
#define TRACE_ADD(role, tile, slot, v)                                                                                    \
    do {                                                                                                                  \
        if (p.trace && blockIdx.x < 4 && (tile) < 64) p.trace[(((int)blockIdx.x * 4 + (role)) * 64 + (tile)) * 8 + (slot)] += (v); \
    } while (0)
#define TRACE_GT(role, tile, slot)                                                                                        \
    do {                                                                                                                  \
        unsigned long long gt_;                                                                                           \
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(gt_));                                                           \
        if (p.trace && blockIdx.x < 4 && (tile) < 64) p.trace[(((int)blockIdx.x * 4 + (role)) * 64 + (tile)) * 8 + (slot)] = (long long)gt_; \
    } while (0)
#else
#define TRACE_GT(role, tile, slot) do {} while (0)
#define TRACE(role, tile, slot) do {} while (0)
#define TRACE_ADD(role, tile, slot, v) do {} while (0)
#endif

struct KParams {
    const int64_t *group_list;
    int gl_len, gl_type;
    int M, K, N;
    int half_n;        // N/2 (swiglu)
    int n_tiles;       // channel tiles per row block
    int max_blocks;    // row blocks that the workspace's counters cover (swiglu)
    int max_tiles;     // their tiles
    int num_k_blocks;  // ceil(K / BK)
    const void *w_nz;     // FRACTAL_NZ weights, read by the loader warps
    const void *w_scale;
    int w_scale_dtype;
    const float *x_scale;
    const void *bias;
    int bias_dtype;
    int act_type, out_f16;
    void *out;            // y (bf16 / int32) or the fp32 SwiGLU staging [M, N/2]
    const long long *out_row_index;  // optional: result row r is written to row out_row_index[r] (bf16 / int32 modes)
    void *out_peers[8];              // bf16 mode with num_peers > 0: out_row_index = (gpu << 40) | row, base per gpu here
    int num_peers;
    // combine epilogue (grouped_matmul_finalize_routing): fp32 result rows added to / stored at row row_index[r] of out
    const float *logit;        // [M] routing weight per row, may be null
    const void *row_index;     // [M] int64 or int32
    int row_index_i32;
    int scatter_add;           // 1: atomic adds (shared-expert rows and logits given), 0: plain stores
    unsigned long long row_limit;  // rows of the result where the caller gave them; indices outside [0, row_limit) are skipped
    unsigned *amax_bits;  // [M] row max of |S| as float bits (swiglu)
    int *rb_counter;      // per row block of a tile two words: arrivals + (hand-overs << 16), and the slice claim counter (swiglu)
    int8_t *q_out;        // int8 [M, N/2] (swiglu)
    float *q_scale_out;   // fp32 [M] (swiglu)
    int *status;
    long long wait_limit;   // cycles a wait may last before the CTA gives up and records kStatusWaitTimeout
    int skip_k_blocks;      // test only: K blocks the producer leaves out of its last tile (drives the abort path)
    int *wave_cnt;          // optional: per wave (round of the static tile schedule) the units that have started it
    int pace_cycles;        // how long a producer waits for the other units to have started the previous wave
#ifdef GMM_TRACE
    long long *trace;
#endif
};

// ---------------------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// CLUSTER: acquires what the other CTA of the pair released (values stored into this CTA's shared memory).
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(WAIT_SUSPEND_NS)
            : "memory");
    else
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(WAIT_SUSPEND_NS)
            : "memory");
    return ok != 0;
}

// The combine's kernel is launched as a programmatic dependent of the one that initialises its result and the status record, and
// runs beside it: everything that it reads was complete before that one started.  Nothing is written to global memory before
// this returns, which is when that kernel has ended and its writes are visible; without such a launch it returns at once.  A warp
// of every CTA also waits before the CTA leaves, whether it had a tile or not: what the stream runs next is ordered behind this
// grid alone, so the grid must not end before the initialisation has.
// (A kernel in the place of every operator's memset would take 2.6 us off a call on the device and cost the host 3.)
__device__ __forceinline__ void wait_for_init() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bounded wait.  Returns false when the limit ran out or another role already gave up.  A change of `*progress` starts the limit
// anew.
template <bool CLUSTER>
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, Shared *sh, int *status, int who,
                                            long long limit, const unsigned *progress = nullptr)
{
    long long t0 = clock64();
    uint32_t spins = 0, seen = 0;
    while (true) {
        if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
        if ((++spins & 31u) == 0u) {
            if (*(volatile int *)&sh->abort_flag) return false;
            const uint32_t now = progress ? *(const volatile unsigned *)progress : 0u;
            if (now != seen) {
                seen = now;
                t0 = clock64();
            }
            if (clock64() - t0 > limit) {
                *(volatile int *)&sh->abort_flag = 1;
                wait_for_init();
                if (atomicCAS(status, kStatusOk, kStatusWaitTimeout) == kStatusOk) {
                    status[1] = (int)blockIdx.x;
                    status[2] = who;
                    status[3] = (int)parity;
                }
                return false;
            }
        }
    }
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, Shared *sh, int *status, int who)
{
    const uint32_t a = smem_u32(bar);
    if (mbar_try_wait<CLUSTER>(a, parity)) return true;
    return mbar_wait_slow<CLUSTER>(a, parity, sh, status, who, sh->wait_limit);
}

// Bounded wait for a work list of swiglu_quant.  Many tiles can lie between two lists - nothing is passed on while none of the
// CTA's row blocks is complete, four blocks times all their channel tiles at a time with few CTAs - and the last list also waits
// for other units (`patience`).  The limit starts anew with every tile that the publishing lane is done with; for each the lane
// waits twice, and bounds these waits itself.
__device__ __forceinline__ bool list_wait(uint64_t *bar, uint32_t parity, Shared *sh, int *status, int who, long long patience)
{
    const uint32_t a = smem_u32(bar);
    if (mbar_try_wait<false>(a, parity)) return true;
    return mbar_wait_slow<false>(a, parity, sh, status, who, 2 * sh->wait_limit + patience, &sh->published);
}

// Tiled TMA loads into this CTA's shared memory.  CTAS == 2 is the pair form: the byte count is credited to the mbarrier at
// `bar`, a shared::cluster address that may belong to the other CTA of the pair.
template <int CTAS>
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint32_t bar)
{
    if (CTAS == 1)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(bar) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar)
{
    if (CTAS == 1)
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                     ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                     ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}
// 16 bytes from global to shared memory, past L1; `bytes` 0 writes zeros without reading.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// One arrival at `bar` (counted in its initial count) when this thread's copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// What was written to shared memory by ordinary accesses and cp.async is visible to the tensor core's reads.
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// L2 eviction policies for the fp32 SwiGLU staging rows: they are read back exactly once, about one tile after they were
// written, while the operands of 74 other tiles stream through L2 in between.  Stored with evict_last and read back with
// evict_first, more of them are still in L2 when they are needed (less DRAM traffic; the time gained is within 1 %).
__device__ __forceinline__ uint64_t policy_evict_first()
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint64_t policy_evict_last()
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void st_global_hint(float *a, float v, uint64_t pol)
{
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(a), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ float4 ld_global_cg_v4_hint(const float4 *a, uint64_t pol)
{
    float4 v;
    asm volatile("ld.global.cg.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(a), "l"(pol) : "memory");
    return v;
}
// One lane of a converged warp.  Copies and MMAs take their operands from uniform registers: issued under this predicate by
// an otherwise converged warp they cost a few cycles each; in a branch that only one thread enters the compiler serialises
// them (about 150 cycles per MMA, which held the whole MMA loop at 600 cycles per K block instead of 512 at 256 tokens).
__device__ __forceinline__ bool elect_one()
{
    uint32_t r;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}
// shared::cluster address of `p` (a location in this CTA's shared memory) as seen in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(const void *p, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
// The same in two parts: what this thread has done and observed in its CTA's shared memory is released to the cluster by the
// next arrival, and an arrival that releases nothing by itself.
__device__ __forceinline__ void fence_release_shared_cluster() { asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t bar_cluster_addr)
{
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ uint32_t cluster_cta_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap *map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <int CTAS>
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t cols)
{
    if (CTAS == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {  // issued by the same warp of both CTAs of the pair, with the same shared-memory offset
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
}
template <int CTAS>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols)
{
    if (CTAS == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem], int8 x int8 -> int32, issued by one thread.
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Pair forms.  The MMA reads A and its half of B from both CTAs' shared memory (same offsets) and writes each CTA's
// 128 accumulator rows to that CTA's TMEM.  The commit takes a shared::cluster address, so it can arrive on a
// barrier of either CTA; it is issued once per CTA of the pair.
__device__ __forceinline__ void umma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// 32 lanes x 32 consecutive columns of 32-bit values: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 16 TMEM lanes x 16 or 32 consecutive columns as matrix fragments: of every 8 columns thread t receives row t/4 in v[4i], v[4i+1]
// and row t/4 + 8 in v[4i+2], v[4i+3], columns 8i + 2 (t%4) and the next one.
__device__ __forceinline__ void tmem_ld16x256b(uint32_t taddr, uint32_t (&v)[8])   // 16 columns
{
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16x256b(uint32_t taddr, uint32_t (&v)[16])   // 32 columns
{
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
// Four 8x8 matrices of 16-bit values, each stored transposed: lane 8j + r names the row of matrix j that receives the
// fragment's column r.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Shared-memory matrix descriptor, version 1.
//   K-major operand : rows of 128 bytes, 8-row groups SBO bytes apart; LBO unused.
//   MN-major operand: runs of one swizzle width along M/N; the next 8 K-rows are SBO bytes on, the next run LBO bytes on.
enum : uint32_t { kSwizzle128 = 2, kSwizzle64 = 4, kSwizzle32 = 6 };
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout_type)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46;
    d |= (uint64_t)layout_type << 61;
    return d;
}

// Descriptor of the weight operand of a stage at `addr`; the next 32 K-rows are weight_k_step bytes on.
template <bool SPLIT, int BL>
__device__ __forceinline__ uint64_t weight_desc(uint32_t addr)
{
    // transposed: rows of 128 K-bytes, one per channel.
    if (BL == kBTransposed) return make_smem_desc(addr, 16, 1024, kSwizzle128);
    // fractal: 32-byte runs along the channels, 8 K-rows = 256 B, next 32 channels 128 K-rows (4096 B) on.
    if (BL == kBFractalNz) return make_smem_desc(addr, 4096, 256, kSwizzle32);
    // [E,K,N], swiglu on a pair: two boxes of 64 channels, 8 K-rows = 512 B, next 64 channels one box on.
    if (SPLIT) return make_smem_desc(addr, W_STAGE / 2, 512, kSwizzle64);
    // [E,K,N]: one box of 128 channels, 8 K-rows = 1024 B.
    return make_smem_desc(addr, W_STAGE, 1024, kSwizzle128);
}
__host__ __device__ constexpr uint32_t weight_k_step(bool split, int bl)
{
    return bl == kBTransposed ? UMMA_K : UMMA_K * (bl == kBFractalNz ? 32u : split ? 64u : 128u);
}

// Instruction descriptor for kind::i8: D = S32 (2 at bit 4), A = B = signed 8-bit (1 at bits 7 and 10), A (weights) major
// per flag (bit 15), B (tokens) K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc(bool a_mn_major, int m)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((uint32_t)(m >> 4) << 24);
}

// ---------------------------------------------------------------------------------------------------------
// Tile schedule, rebuilt by every CTA from group_list (<= 1024 entries)
// ---------------------------------------------------------------------------------------------------------

// Row blocks of a group of `rows` rows, as few as MAX_TOK rows a tile allow, and the token rows of each: of nearly equal size
// (a multiple of 32; no more than MAX_TOK, so the count stays the same).  Equal tiles keep the units of a wave together; their
// sum costs the same as full tiles and a short one.
template <int MAX_TOK>
__device__ __forceinline__ int row_blocks(int rows) { return (rows + MAX_TOK - 1) / MAX_TOK; }
template <int MAX_TOK>
__device__ __forceinline__ int tile_tokens(int rows)
{
    const int nt = row_blocks<MAX_TOK>(rows);
    const int each = nt <= 1 ? max(rows, 1) : (rows + nt - 1) / nt;   // (no division on the way of a short call)
    return (each + TOK_STEP - 1) / TOK_STEP * TOK_STEP;
}

// Row ranges follow GetSplitValueFromGroupList (gmm/grouped_matmul/op_kernel/grouped_matmul_utils.h:243-257):
// type 0 = running total, type 1 = count, values narrowed to int32; groups with no rows are skipped
// (grouped_matmul.h:263).  Ranges are clipped to [0, M] so a malformed list cannot address other memory.  Disjoint ranges have
// at most ceil(M / 128) + L row blocks; a falling running total names rows again and again and can have many times as many.  The
// swiglu tiles beyond the counters reserved for that many are left out and reported (kStatusBadList): the counters behind them
// are other data, and a slice claimed from such a word would be an arbitrary range of rows.
//
// The last wave: `rem` tiles for n_units units take as long as a full wave.  Where two or more units are there for each of
// them, they are cut into that many pieces along their tokens: the weights come from L2 for all but one of the pieces.  The
// number of pieces is one for the launch, no more than bring its largest tile down to SPLIT_TOK (below, a K block of MMAs does
// not get shorter any more); smaller tiles get pieces of a multiple of 32 tokens, and one without rows is left out.  (Pieces of at
// least SPLIT_TOK whatever the tile take the same time within the runs' spread: K=7168 N=2048, 256 rows and five groups of 100, us
// as here / so: grouped_matmul 32.0 / 32.8, swiglu_quant 38.5 / 38.5.)
// K=4096 N=4096, 6 groups of about 200 rows, us: grouped_matmul 32.9 -> 31.1, swiglu_quant 40.2 -> 38.5.
template <int MAX_TOK>
__device__ void build_schedule(Shared *sh, const KParams &p, int n_units)
{
    const int tid = threadIdx.x, L = p.gl_len;
    for (int g = tid; g < L; g += (int)blockDim.x) {
        const int v = (int)p.group_list[g];
        int start = 0, rows = v;
        if (p.gl_type == 0) {
            const int prev = g ? (int)p.group_list[g - 1] : 0;
            start = prev;
            rows = v - prev;
        }
        sh->row_start[g] = start;
        sh->rows[g] = rows;
    }
    __syncthreads();
    if (tid < 32) {
        const int lane = tid;
        const int chunk = (L + 31) / 32;
        const int lo = min(lane * chunk, L), hi = min(lo + chunk, L);
        if (p.gl_type != 0) {
            int s = 0;
            for (int g = lo; g < hi; ++g) s += max(sh->rows[g], 0);
            int incl = s;
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += n;
            }
            int run = incl - s;
            for (int g = lo; g < hi; ++g) {
                sh->row_start[g] = run;
                run += max(sh->rows[g], 0);
            }
        }
        int tsum = 0, max_tok = TOK_STEP;
        for (int g = lo; g < hi; ++g) {
            long long start = sh->row_start[g], rows = sh->rows[g];
            if (rows < 0) rows = 0;
            if (start < 0) { rows += start; start = 0; if (rows < 0) rows = 0; }
            if (start > p.M) { start = p.M; rows = 0; }
            if (start + rows > p.M) rows = p.M - start;
            sh->row_start[g] = (int)start;
            sh->rows[g] = (int)rows;
            const int tt = tile_tokens<MAX_TOK>((int)rows);
            const int tiles = row_blocks<MAX_TOK>((int)rows) * p.n_tiles;
            max_tok = max(max_tok, tt);
            sh->tile_start[g] = tiles;
            tsum += tiles;
        }
        int incl = tsum;
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        int run = incl - tsum;
        for (int g = lo; g < hi; ++g) {
            const int tiles = sh->tile_start[g];
            sh->tile_start[g] = run;
            run += tiles;
        }
        max_tok = __reduce_max_sync(0xffffffffu, max_tok);
        if (lane == 31) {
            sh->max_tok = max_tok;
            sh->tile_start[L] = incl;
            const int total = min(incl, p.max_tiles), rem = total < n_units ? total : total % n_units;
            int split = max_tok > SPLIT_TOK && rem > 0 ? min(n_units / rem, (max_tok + SPLIT_TOK - 1) / SPLIT_TOK) : 1;
            if (split < 2 || p.n_tiles > 32767 / (2 * split)) split = 1;   // shares of a row block are counted in 16 bits
            sh->split = split;
            sh->split_from = split > 1 ? total - rem : total;
            sh->total_tiles = split > 1 ? total - rem + rem * split : total;
            if (incl > p.max_tiles && blockIdx.x == 0 && atomicCAS(p.status, kStatusOk, kStatusBadList) == kStatusOk) {
                p.status[1] = 0;
                p.status[2] = 810;
                p.status[3] = L;
            }
        }
    }
    __syncthreads();
}

// Rows of x a CTA loads per K block for its share of a tile: one box, the smallest of 32, 64 or 128 rows that covers the
// share, or two of 128.
template <int CTAS>
__device__ __forceinline__ int x_box_rows(int share)
{
    return CTAS == 1 && share > 128 ? 256 : share > 64 ? 128 : share > 32 ? 64 : 32;
}

// Token rows of each piece of a tile of `rows` rows cut into `split` (the last one may have fewer, or none).
__device__ __forceinline__ int piece_tokens(int rows, int split)
{
    return ((rows + split - 1) / split + TOK_STEP - 1) / TOK_STEP * TOK_STEP;
}

struct Tile {
    int g, row0, rows, n_idx;           // rows <= 0: a piece without rows, always a unit's last one
    int index, block_row0, block_rows;  // of the whole tile
    int block, block_last;              // its row block, and the last tile of that
};

// `from`: the group of this unit's previous tile (tiles are visited in ascending order); normally the next one is near.
template <int MAX_TOK, int BLOCK_GROUP>
__device__ __forceinline__ Tile decode_tile(const Shared *sh, int t, int n_tiles, int L, int from = 0)
{
    int piece = -1;
    if (t >= sh->split_from) {
        const int v = t - sh->split_from, k = v / sh->split;
        piece = v - k * sh->split;
        t = sh->split_from + k;
    }
    int lo = from, hi = min(from + 4, L);  // largest g in [0, L) with tile_start[g] <= t
    if (sh->tile_start[hi] <= t) { lo = hi; hi = L; }
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sh->tile_start[mid] <= t) lo = mid; else hi = mid;
    }
    // BLOCK_GROUP row blocks of a group at a time; of them all row blocks of a channel tile, then the next channel tile
    const int rows = sh->rows[lo], local = t - sh->tile_start[lo], per = BLOCK_GROUP * n_tiles;
    const int sg = local < per ? 0 : local / per, rem = local - sg * per;
    const int side = min(BLOCK_GROUP, row_blocks<MAX_TOK>(rows) - sg * BLOCK_GROUP);
    const int tt = tile_tokens<MAX_TOK>(rows);
    Tile tl;
    tl.g = lo;
    tl.n_idx = side == 1 ? rem : rem / side;
    const int in_side = rem - tl.n_idx * side, mb = sg * BLOCK_GROUP + in_side;
    tl.row0 = sh->row_start[lo] + mb * tt;
    tl.rows = min(tt, rows - mb * tt);
    tl.block = sh->tile_start[lo] / n_tiles + mb;
    tl.block_last = sh->tile_start[lo] + sg * per + (n_tiles - 1) * side + in_side;
    tl.index = t;
    tl.block_row0 = tl.row0;
    tl.block_rows = tl.rows;
    if (piece >= 0) {
        const int sub = piece_tokens(tl.rows, sh->split);
        tl.row0 += piece * sub;
        tl.rows = min(sub, tl.rows - piece * sub);
    }
    return tl;
}

// ---------------------------------------------------------------------------------------------------------
// Epilogue helpers
// ---------------------------------------------------------------------------------------------------------

__device__ __forceinline__ float load_scale1(const void *p, int dtype, size_t i)
{
    if (dtype == kF32) return __ldg(reinterpret_cast<const float *>(p) + i);
    const uint16_t h = __ldg(reinterpret_cast<const uint16_t *>(p) + i);
    if (dtype == kBF16) return __uint_as_float((uint32_t)h << 16);
    return __half2float(__ushort_as_half(h));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // one cvt.rn.bf16x2.f32, round to nearest even
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi)
{
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// Four fp32 additions to 16 aligned bytes of global memory in one request, no value returned.
__device__ __forceinline__ void red_add_v4(float *p, const float4 v)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// q = int8(rint(half(S * (1 / (amax / 127)))))  -- CastFp32ToInt8Template,
// gmm/grouped_matmul_swiglu_quant/op_kernel/grouped_matmul_swiglu_quant_utils.h:308-316; NaN -> 0, saturating.
__device__ __forceinline__ uint32_t quant1(float s, float rcp)
{
    const __half h = __float2half_rn(__fmul_rn(s, rcp));
    const int q = max(-128, min(127, __half2int_rn(h)));
    return (uint32_t)q & 0xffu;
}
__device__ __forceinline__ uint32_t quant4(float4 v, float rcp)
{
    return quant1(v.x, rcp) | (quant1(v.y, rcp) << 8) | (quant1(v.z, rcp) << 16) | (quant1(v.w, rcp) << 24);
}
// The same for a row whose scale lies in [1e-30, 1e30]: no finite value leaves [-127, 127], so nothing saturates, and adding
// 1536 to the fp16 value rounds it to the nearest integer (ties to even: the spacing there is 1) and leaves that integer in the
// low byte.  NaN, which the row maximum left out, becomes 0.
__device__ __forceinline__ uint32_t quant4_plain(float4 v, f32x2 rcp)
{
    const float2 a = unpair2(mul2(pair2(v.x, v.y), rcp)), b = unpair2(mul2(pair2(v.z, v.w), rcp));
    const __half2 ha = __floats2half2_rn(a.x, a.y), hb = __floats2half2_rn(b.x, b.y);
    const __half2 magic = __halves2half2(__ushort_as_half(0x6600), __ushort_as_half(0x6600));
    const __half2 qa = __hadd2(ha, magic), qb = __hadd2(hb, magic);
    return __byte_perm(*reinterpret_cast<const uint32_t *>(&qa) & __heq2_mask(ha, ha),
                       *reinterpret_cast<const uint32_t *>(&qb) & __heq2_mask(hb, hb), 0x6420);
}

// Second half of grouped_matmul_swiglu_quant for rows [r_begin, r_end) of a finished row block (all of its N tiles
// have stored S and the row maxima): per row  qs = amax / 127, r = 1 / qs, q = int8(half(S * r))
// (gmm/grouped_matmul_swiglu_quant/op_kernel/grouped_matmul_swiglu_quant.h:496-503).  S and amax were written by
// other SMs, so they are read through L2 (ld.global.cg).  One warp per row.  Consecutive lanes read consecutive 16-byte
// pieces (a load instruction covers 512 contiguous bytes, a store 128): the tensor cores read their operands through the
// same shared-memory / L1 data path, so every extra line these accesses touch is taken from the MMAs.  Sixteen loads
// per lane are in flight at a time, because they wait for L2 under the full load of the GEMM.
// Not inlined: the epilogue warps take part in the last list, and a second copy would only have to be fetched again.  With their
// help, without empty lists and with fewer instructions per value, the end of a short call got shorter: K=4096 N=4096, 6 groups
// of about 200 rows 41.6 -> 40.2 us, K=1408 N=1408, 22 groups of 12 rows 22.5 -> 21.9.
__device__ __noinline__ void requant_rows(const float *stage, const unsigned *amax_bits, int8_t *q_out, float *q_scale_out, int H, int r_begin,
                                          int r_end, int worker, int workers)
{
    const int lane = threadIdx.x & 31;
    const int nf = H >> 2;  // 16-byte pieces per row
    const uint64_t pol_first = policy_evict_first();
    for (int grow = r_begin + worker; grow < r_end; grow += workers) {
        const float amax = __uint_as_float(__ldcg(amax_bits + grow));
        const float4 *src = reinterpret_cast<const float4 *>(stage + (size_t)grow * H);
        uint32_t *dst = reinterpret_cast<uint32_t *>(q_out + (size_t)grow * H);
        for (int f = lane; f - lane < nf; f += 512) {
            float4 v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = f + 32 * u < nf ? ld_global_cg_v4_hint(src + f + 32 * u, pol_first) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float qs = __fdiv_rn(amax, 127.0f);
            const float rcp = __fdiv_rn(1.0f, qs);
            if (f == 0) q_scale_out[grow] = qs;
            if (qs >= 1e-30f && qs <= 1e30f) {
                const f32x2 rcp2 = pair2(rcp, rcp);
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (f + 32 * u < nf) dst[f + 32 * u] = quant4_plain(v[u], rcp2);
            } else {
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (f + 32 * u < nf) dst[f + 32 * u] = quant4(v[u], rcp);
            }
        }
    }
}

// Who requantises a finished row block, without any CTA ever waiting for another one (so the kernel does not depend on
// all CTAs being resident at the same time, nor on how many there are).
//
// Per row block two words in the workspace: state = arrivals (low 16 bits) + handed-over shares (high 16 bits), and a
// claim counter.  A block has `shares` contributors (N tiles x CTAs per tile) and is requantised in `shares` row slices.
//   * A CTA that has stored its part of the block "arrives" (atomic add of 1 after a fence).  The arrival that completes
//     the block takes one slice for itself plus one for every share handed over so far.
//   * Every other contributor keeps the block on a short pending list and looks at the state again after each of its
//     later tiles; once the block is complete it takes one slice.
//   * A contributor that cannot come back (its last tile is done, or its list is full) hands its share over with an
//     atomic add of 1 << 16.  If that add finds the block already complete it takes its slice itself; otherwise the
//     completing arrival, which comes later, sees the hand-over in the value its own add returns.
// Slices are claimed from the claim counter, so every slice is taken exactly once.
__device__ __forceinline__ void add_work(Shared *sh, int ws, const PendingBlock &b, int first, int count)
{
    const int k = sh->n_work[ws]++;
    sh->work_begin[ws][k] = b.row0 + (int)((long long)b.rows * first / b.shares);
    sh->work_end[ws][k] = b.row0 + (int)((long long)b.rows * (first + count) / b.shares);
}

// This CTA's shares of block `b` go to whoever completes it, or are taken now if that has happened.
__device__ __forceinline__ void hand_over(const KParams &p, Shared *sh, int ws, const PendingBlock &b)
{
    const int o = atomicAdd(p.rb_counter + 2 * b.rb, b.weight << 16);
    if ((o & 0xffff) == b.shares) add_work(sh, ws, b, atomicAdd(p.rb_counter + 2 * b.rb + 1, b.weight), b.weight);
}

__device__ __forceinline__ int ld_relaxed_gpu(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Publishing lane, after the whole CTA has stored a tile: arrive at its block, look at the pending blocks, fill work list
// `ws`.  The caller fences before (release of the CTA's stores) and after (acquire of the other CTAs' stores).
__device__ void publish_and_collect(const KParams &p, Shared *sh, int ws, const PendingBlock &mine)
{
    int *state = p.rb_counter;
    // the looks at the older blocks and the arrival travel together (one round trip to L2)
    int seen[MAX_PENDING];
#pragma unroll
    for (int i = 0; i < MAX_PENDING; ++i) seen[i] = i < sh->pend_n ? ld_relaxed_gpu(state + 2 * sh->pend[i].rb) : 0;
    const int old = atomicAdd(state + 2 * mine.rb, mine.weight);
    const bool completed = (old & 0xffff) + mine.weight == mine.shares;
    // slice claims, again together
    int first[MAX_PENDING];
#pragma unroll
    for (int i = 0; i < MAX_PENDING; ++i)
        first[i] = (i < sh->pend_n && (seen[i] & 0xffff) == sh->pend[i].shares) ? atomicAdd(state + 2 * sh->pend[i].rb + 1, sh->pend[i].weight) : -1;
    const int cnt = mine.weight + (old >> 16);
    const int my_first = completed ? atomicAdd(state + 2 * mine.rb + 1, cnt) : -1;
    int n = 0;
#pragma unroll
    for (int i = 0; i < MAX_PENDING; ++i) {
        if (i >= sh->pend_n) break;
        if (first[i] >= 0) add_work(sh, ws, sh->pend[i], first[i], sh->pend[i].weight);
        else sh->pend[n++] = sh->pend[i];
    }
    sh->pend_n = n;
    if (completed) {
        add_work(sh, ws, mine, my_first, cnt);
        return;
    }
    if (sh->pend_n == MAX_PENDING) {  // hand the oldest block's share over (or take it, if the block completed meanwhile)
        hand_over(p, sh, ws, sh->pend[0]);
        for (int i = 1; i < MAX_PENDING; ++i) sh->pend[i - 1] = sh->pend[i];
        --sh->pend_n;
    }
    sh->pend[sh->pend_n++] = mine;
}

// Publishing lane, after the CTA's last tile: every block still pending is taken once it is complete.  The other units
// are finishing at the same time, so the lane first looks on for up to `patience` cycles (nothing else is left to do;
// handing the share over at once would leave the last arrival of every block of the final wave with all of its slices,
// a serial tail of tens of microseconds); what is still incomplete after that is handed over, so the kernel never
// depends on the other CTAs being resident.
__device__ void release_pending(const KParams &p, Shared *sh, int ws, long long patience)
{
    int *state = p.rb_counter;
    const long long t0 = clock64();
    while (sh->pend_n > 0) {
        int n = 0;
        for (int i = 0; i < sh->pend_n; ++i) {
            if ((ld_relaxed_gpu(state + 2 * sh->pend[i].rb) & 0xffff) == sh->pend[i].shares)
                add_work(sh, ws, sh->pend[i], atomicAdd(state + 2 * sh->pend[i].rb + 1, sh->pend[i].weight), sh->pend[i].weight);
            else sh->pend[n++] = sh->pend[i];
        }
        sh->pend_n = n;
        if (n == 0 || clock64() - t0 > patience) break;
        __nanosleep(100);
    }
    for (int i = 0; i < sh->pend_n; ++i) hand_over(p, sh, ws, sh->pend[i]);
    sh->pend_n = 0;
}

// The row ranges of work list `ws`, which the caller has acquired: worker w of n takes rows w, w + n, ... of each.
__device__ __forceinline__ void work_off(const KParams &p, const Shared *sh, int ws, int worker, int workers)
{
    const int n = sh->n_work[ws];
    for (int k = 0; k < n; ++k)
        requant_rows(static_cast<const float *>(p.out), p.amax_bits, p.q_out, p.q_scale_out, p.half_n, sh->work_begin[ws][k], sh->work_end[ws][k], worker, workers);
}

// v / (1 + exp(-z)), for z < 0 as v e / (1 + e), with e = exp(-|z|) so that nothing overflows.
//   e = 2^t (1 + d ln 2): t is the rounded product -|z| h of h = fl(log2 e), d = -|z| (h + l) - t what the rounding and the
//   remainder l of log2 e = h + l left out (an fma each; |d| < 2^-16, so the second-order term is below 2^-33).
//   The quotient comes from an approximate reciprocal r of the denominator in [1, 2] and one correction q + (n - q den) r
//   (Markstein, IA-64 and Elementary Functions, 2000).
// Below z = -64, where 1 + e is 1, e is kept multiplied by 4 until the last step: the flush of ex2 to zero then begins at
// 2^-128, which is where 1 + expf(-z) of apply_activation overflows and its quotient becomes zero; unscaled it began at 2^-126
// and took the results for z in [-88.72, -87.34] (about 5e-37) with it.
// Error: ex2 2 ulp, its correction, n, the denominator, the quotient and its correction a rounding each: below 4 ulp of the
// exact value down to the point where it vanishes, like expf and a division rounded once (which also sees expf's 2 ulp).  The
// two differ in the last places, so the SIMT kernels' results (apply_activation) are not bit for bit the same.
// An infinite quotient is kept as it is; NaN stays NaN.
__device__ __forceinline__ float times_sigmoid(float v, float z)
{
    const bool tail = z < -64.0f;
    const float x = fminf(fabsf(z), 150.0f);
    float t = __fmul_rn(x, -1.44269502f);
    const float d = __fmaf_rn(x, -1.92596299e-8f, __fmaf_rn(x, -1.44269502f, -t));
    if (tail) t = __fadd_rn(t, 2.0f);   // exact: |t| > 92
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
    e = __fmaf_rn(e, __fmul_rn(d, 0.693147181f), e);
    const float den = __fadd_rn(1.0f, e);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(den));
    const float n = z < 0.0f ? __fmul_rn(v, e) : v;
    const float q = __fmul_rn(n, r);
    const float c = __fmaf_rn(__fmaf_rn(-q, den, n), r, q);
    const float res = fabsf(q) <= 3.402823466e38f ? c : q;
    return tail ? __fmul_rn(res, 0.25f) : res;
}

// The same for two values with |z| <= kPlainZ: exp(-z) stays between 2^-93 and 2^93, so neither a sign nor the range has to be
// looked at, and v / (1 + exp(-z)) is formed as it stands: 9 packed instructions and two approximations each instead of twice
// 20 instructions.  The error is that of times_sigmoid less the rounding of v e.  (K=1024 N=2048, 64 groups of 400 rows: swiglu
// 118 -> 115 us; K=1424 N=2976, 3055 rows, fp16 with bias and GELU: 41 -> 39.)
constexpr float kPlainZ = 64.0f;
__device__ __forceinline__ f32x2 times_sigmoid2(f32x2 v, f32x2 z)
{
    const f32x2 log2e = pair2(1.44269502f, 1.44269502f), neg_log2e = pair2(-1.44269502f, -1.44269502f);
    const f32x2 t = mul2(z, log2e);   // the exponent is -t
    const f32x2 d = fma2(z, pair2(-1.92596299e-8f, -1.92596299e-8f), fma2(z, neg_log2e, t));
    const float2 ts = unpair2(t);
    float e0, e1, r0, r1;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(-ts.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(-ts.y));
    f32x2 e = pair2(e0, e1);
    e = fma2(e, mul2(d, pair2(0.693147181f, 0.693147181f)), e);
    const f32x2 minus1 = pair2(-1.0f, -1.0f);
    const f32x2 neg_den = fma2(e, minus1, minus1);
    const float2 nd = unpair2(neg_den);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-nd.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-nd.y));
    const f32x2 r = pair2(r0, r1), q = mul2(v, r);
    return fma2(fma2(q, neg_den, v), r, q);
}

// Over a thread's N values: the short form where z allows it, so that a result does not depend on what is computed beside it,
// and nothing else where the whole warp's z do, as those of a layer.
template <int N>
__device__ __forceinline__ void times_sigmoids(float (&v)[N], const float (&z)[N])
{
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) m = fmaxf(m, fabsf(z[i]));
    if (__all_sync(0xffffffffu, m <= kPlainZ)) {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const float2 r = unpair2(times_sigmoid2(pair2(v[i], v[i + 1]), pair2(z[i], z[i + 1])));
            v[i] = r.x;
            v[i + 1] = r.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const float2 r = unpair2(times_sigmoid2(pair2(v[i], v[i + 1]), pair2(z[i], z[i + 1])));
            v[i] = fabsf(z[i]) <= kPlainZ ? r.x : times_sigmoid(v[i], z[i]);
            v[i + 1] = fabsf(z[i + 1]) <= kPlainZ ? r.y : times_sigmoid(v[i + 1], z[i + 1]);
        }
    }
}

// apply_activation (gmm_common.h) over a thread's values, the choice made once: with a switch in every element the unrolled
// epilogue was several thousand instructions long and ran out of the instruction cache (3055 x 2976, K = 1424, fp16: 58 us
// without an activation and 95 us with GELU, against 30 us for the instance without options).
template <int N>
__device__ __forceinline__ void activate(int act_type, float (&v)[N])
{
    if (act_type == 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = v[i] > 0.0f ? v[i] : 0.0f;
    } else if (act_type == 2) {   // z = 1.596 (v + 0.0447 v^3); its sum has one rounding fewer here than in apply_activation
        float z[N];
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const f32x2 x = pair2(v[i], v[i + 1]);
            const f32x2 x3 = mul2(mul2(x, x), x);
            const float2 zi = unpair2(mul2(pair2(1.59576912f, 1.59576912f), fma2(pair2(0.044715f, 0.044715f), x3, x)));
            z[i] = zi.x;
            z[i + 1] = zi.y;
        }
        times_sigmoids(v, z);
    } else if (act_type == 4 || act_type == 5) {
        const float f = act_type == 4 ? 1.702f : 1.0f;
        float z[N];
#pragma unroll
        for (int i = 0; i < N; ++i) z[i] = __fmul_rn(f, v[i]);
        times_sigmoids(v, z);
    }
}

// (acc * x_scale) * w_scale of one channel's 16 tokens; `tok` is 16-byte aligned.
__device__ __forceinline__ void dequant16(const uint32_t (&acc)[16], const float *tok, float w_scale, float (&out)[16])
{
    const f32x2 w = pair2(w_scale, w_scale);
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(tok + i);
        const float2 lo = unpair2(mul2(mul2(pair2(__int2float_rn((int)acc[i]), __int2float_rn((int)acc[i + 1])), pair2(x.x, x.y)), w));
        const float2 hi = unpair2(mul2(mul2(pair2(__int2float_rn((int)acc[i + 2]), __int2float_rn((int)acc[i + 3])), pair2(x.z, x.w)), w));
        out[i] = lo.x; out[i + 1] = lo.y; out[i + 2] = hi.x; out[i + 3] = hi.y;
    }
}
// S = gate * (act / (1 + exp(-act))), into act
__device__ __forceinline__ void swiglu16(float (&act)[16], const float (&gate)[16])
{
    float z[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) z[i] = act[i];
    times_sigmoids(act, z);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const float2 r = unpair2(mul2(pair2(gate[i], gate[i + 1]), pair2(act[i], act[i + 1])));
        act[i] = r.x;
        act[i + 1] = r.y;
    }
}

// A meeting of the epilogue warps that exchange values through shared memory (2 or 4 of them per barrier): every warp's
// earlier accesses to the staging area are done and visible to the others when it returns.  Bounded like every wait, and
// the same answer for all lanes of a warp; false = give up.
__device__ __forceinline__ bool group_sync(uint64_t *bar, uint32_t &phase, Shared *sh, int *status, int lane, int who)
{
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
    const bool ok = mbar_wait(bar, phase, sh, status, who);
    phase ^= 1u;
    return __all_sync(0xffffffffu, ok);
}

// 16 tokens x 32 channels of 32-bit values, one channel per lane: afterwards eight lanes hold 128 contiguous bytes of one
// token's row.  Piece i of lane l is token i * 4 + l / 8, channels 4 * (l % 8) .. + 3.
__device__ __forceinline__ void transpose16(uint8_t *stage, const uint32_t (&v)[16], int lane, uint4 (&out)[4])
{
#pragma unroll
    for (int t = 0; t < 16; ++t) *reinterpret_cast<uint32_t *>(stage + t * 128 + lane * 4) = v[t];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = *reinterpret_cast<const uint4 *>(stage + (i * 4 + (lane >> 3)) * 128 + (lane & 7) * 16);
    __syncwarp();
}

// ---------------------------------------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------------------------------------

struct XMaps {
    CUtensorMap box[X_MAPS];  // boxes of 32 << i rows
};

// EPI selects the epilogue variant: kEpiPlain = no bias, no activation, rows stored in place (the common case, compiled without
// per-element tests for the options); kEpiScatter = the same arithmetic with the result rows scattered through out_row_index,
// optionally into other GPUs' memory; kEpiHalf, kEpiHalfScatter = the same two for fp16 results; kEpiCombine = fp32 rows added
// into row_index; kEpiGeneric = bias or activation, every option tested at run time.  CTAS: 1 = one CTA per tile (128 channels), 2 = a cluster of two CTAs (256 channels).
template <int MODE, int BL, int EPI, int CTAS>
__global__ void __launch_bounds__(num_threads(MODE, BL, EPI), 1)
gmm_w8a8_sm100_kernel(const __grid_constant__ XMaps maps_x, const __grid_constant__ CUtensorMap map_w, const KParams p)
{
    constexpr bool PLAIN = EPI != kEpiGeneric;   // lean arithmetic
    constexpr bool SCATTER = EPI != kEpiPlain && EPI != kEpiHalf;  // rows go where out_row_index says
    constexpr bool COMBINE = EPI == kEpiCombine;  // fp32 rows combined into row_index[r] of a [out_rows, N] result
    constexpr bool SWIGLU = MODE == kModeSwigluQuant;
    constexpr bool OUT16 = MODE == kModeDequantBf16 && !COMBINE;
    using S = Shape<MODE, CTAS>;
    constexpr bool NZ = BL == kBFractalNz;       // weights come through the loader warps
    constexpr int EPI_WARPS = epi_warps(MODE, EPI), EPI_THREADS = 32 * EPI_WARPS, CHUNK = chunk_tokens(MODE, EPI);
    constexpr int RQ = rq_warps(BL), LD0 = num_threads(MODE, BL, EPI) / 32 - ld_warps(BL);   // first loader warp
    constexpr bool DUAL = S::kDual;
    constexpr int CH_CTA = S::kCols, MAX_TOK = S::kMaxTok, W_BYTES = S::kWStage;
    constexpr int BLOCK_GROUP = block_group(MODE);
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    Shared *sh = reinterpret_cast<Shared *>(smem + PIPE_BYTES);
    // stage s: this CTA's channels at smem + s * stage_bytes, its token rows right behind them

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // known to be uniform
    const uint32_t rank = CTAS == 2 ? cluster_cta_rank() : 0u;  // position in the pair; rank 0 issues the MMAs
    const int unit = CTAS == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;   // tile-processing unit (CTA or pair)
    const int n_units = CTAS == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            // The producer arrives once and the copies credit their bytes (pair: at rank 0's barrier, for both CTAs); loader
            // threads arrive each at their own CTA's barrier, and rank 1's, complete, is passed on to rank 0 as one more.
            mbar_init(&sh->full[s], !NZ ? 1 : rank == 0 ? 32 * LD_WARPS + CTAS : 32 * LD_WARPS);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            // one arrival per epilogue warp of this CTA; pair: rank 1's, complete, is passed on to rank 0 as one more
            mbar_init(&sh->acc_empty[b], EPI_WARPS + (CTAS == 2 && rank == 0 ? 1 : 0));
            mbar_init(&sh->tok_ready[b], EPI_THREADS);
        }
        for (int b = 0; b < 4; ++b) mbar_init(&sh->grp_sync[b], SWIGLU ? 2 : 4);
        for (int b = 0; b < WK_DEPTH; ++b) {
            mbar_init(&sh->wk_full[b], 1);
            mbar_init(&sh->wk_empty[b], RQ);
        }
        mbar_init(&sh->wk_closing, 1);
        sh->stored_count = 0;
        sh->published = 0;
        sh->abort_flag = 0;
        sh->total_tiles = 0;
        sh->wait_limit = p.wait_limit;
        sh->pend_n = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < X_MAPS; ++i) prefetch_map(&maps_x.box[i]);
        prefetch_map(&map_w);
    }
    if (warp == 1) {
        tmem_alloc<CTAS>(&sh->tmem_base, TMEM_COLS);
        tc_fence_before();
    }
    build_schedule<MAX_TOK>(sh, p, n_units);  // ends with __syncthreads()
    if (CTAS == 2) cluster_sync_all();  // the partner's barriers exist before anything is sent to them
    tc_fence_after();

    const int total_tiles = sh->total_tiles;
    const int stage_bytes = W_BYTES + x_box_rows<CTAS>(sh->max_tok / CTAS) * BK;
    const int stages = min(PIPE_BYTES / stage_bytes, MAX_STAGES);
    const uint32_t tmem_base = sh->tmem_base;
    const int L = p.gl_len;

    if (CTAS == 2 && rank == 1 && warp == (NZ ? 0 : 1)) {
        // ------------------------------ rank 1, a warp without other work: its epilogue's releases to rank 0 ------------------------------
        // An arrival at the other CTA's barrier with cluster-wide release takes 1450 cycles; here no epilogue warp waits for it.
        const uint32_t acc_empty_rank0 = map_to_cta(&sh->acc_empty[0], 0);
        int buf = 0;
        uint32_t acc_phase = 0;
        for (int t = unit; t < total_tiles; t += n_units) {
            if (t >= sh->split_from && decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t, p.n_tiles, L).rows <= 0) break;
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_empty[buf], acc_phase, sh, p.status, 210 + buf))) break;
            tc_fence_after();
            tc_fence_before();
            if (lane == 0) mbar_arrive_cluster(acc_empty_rank0 + (uint32_t)buf * 8u);
            __syncwarp();
            buf ^= 1;
            if (buf == 0) acc_phase ^= 1u;
        }
    } else if (warp == 0) {
        // ------------------------------ TMA producer (whole warp, one elected lane issues) ------------------------------
        {
            const bool leader = elect_one();
            int stage = 0;
            uint32_t phase = 0;
            long long issued = 0;
            bool ok = true;
            // pair: rank 0's full barriers as shared::cluster addresses (barriers are 8 bytes apart)
            const uint32_t full_rank0 = CTAS == 2 ? map_to_cta(&sh->full[0], 0) : 0u;
            // Pacing: the units of a wave (one round of the static schedule) share their operands through L2 - the channel
            // tiles of a row block read the same rows of x, the row blocks of an expert the same weight boxes - and one launch
            // streams many times the L2's capacity, so a unit that drifts a tile or two away from the others finds the
            // shared data evicted and fetches it from DRAM again.  Every unit therefore announces the wave it starts and
            // waits, for at most about one tile's duration, until all units have started the wave before.  It is a hint,
            // never needed for correctness: when the wait runs out (units not resident together) pacing is switched off.
            bool pace = p.wave_cnt != nullptr && rank == 0;
            int wave = 0;
            Tile next = unit < total_tiles ? decode_tile<MAX_TOK, BLOCK_GROUP>(sh, unit, p.n_tiles, L) : Tile{};
            for (int t = unit; t < total_tiles && ok; t += n_units, ++wave) {
                const Tile tl = next;
                if (tl.rows <= 0) break;
                if (pace) {
                    if (lane == 0) {
                        if (wave > 0) {
                            const int expected = min(n_units, total_tiles - (wave - 1) * n_units);
                            const long long t0 = clock64();
                            while (ld_relaxed_gpu(p.wave_cnt + wave - 1) < expected) {
                                if (clock64() - t0 > p.pace_cycles) { pace = false; break; }
                                __nanosleep(500);
                            }
                        }
                        asm volatile("red.relaxed.gpu.global.add.s32 [%0], 1;" ::"l"(p.wave_cnt + wave) : "memory");
                    }
                    pace = __shfl_sync(0xffffffffu, pace ? 1 : 0, 0) != 0;
                }
                // This CTA's share of the tokens; rows beyond the group or the tensor (zero filled) are never stored.
                const int my_tok = (tl.rows + TOK_STEP - 1) / TOK_STEP * TOK_STEP / CTAS;
                const int my_row0 = tl.row0 + (int)rank * my_tok;
                const int x_rows = x_box_rows<CTAS>(my_tok);
                const CUtensorMap *map_x = &maps_x.box[x_rows >= 128 ? 2 : x_rows >= 64 ? 1 : 0];
                const uint32_t tx_bytes = (uint32_t)CTAS * (uint32_t)((NZ ? 0 : W_BYTES) + x_rows * BK);
                const int c0 = (tl.n_idx * CTAS + (int)rank) * CH_CTA;   // first weight column of this CTA
                // test hook: leaving K blocks out of the last tile makes the MMA issuer's wait run out (nothing else is touched)
                const int kb_end = p.num_k_blocks - (t + n_units >= total_tiles ? p.skip_k_blocks : 0);
                for (int kb = 0; kb < kb_end; ++kb) {
#ifdef GMM_TRACE
                    const long long tw0 = clock64();
#endif
                    if (!__all_sync(0xffffffffu, mbar_wait(&sh->empty[stage], phase ^ 1u, sh, p.status, 100 + stage))) { ok = false; break; }
#ifdef GMM_TRACE
                    if (lane == 0) TRACE_ADD(0, wave, 2, clock64() - tw0);
#endif
                    if (leader) {
                        uint8_t *wdst = smem + stage * stage_bytes;
                        const uint32_t bar = CTAS == 2 ? full_rank0 + (uint32_t)stage * 8u : smem_u32(&sh->full[stage]);
                        if (rank == 0) mbar_arrive_expect_tx(&sh->full[stage], tx_bytes);
                        if (BL == kBTransposed) tma_load_4d<CTAS>(wdst, &map_w, kb * BK, c0, 0, tl.g, bar);
                        else if (!NZ) tma_load_4d<CTAS>(wdst, &map_w, c0, kb * BK, 0, tl.g, bar);
                        tma_load_2d<CTAS>(wdst + W_BYTES, map_x, kb * BK, my_row0, bar);
                        if (CTAS == 1 && x_rows > 128) tma_load_2d<CTAS>(wdst + W_BYTES + 128 * BK, map_x, kb * BK, my_row0 + 128, bar);
                    }
                    __syncwarp();
                    // the next tile is looked up while the ring is full, not between two tiles
                    if (kb == 0 && t + n_units < total_tiles) next = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t + n_units, p.n_tiles, L, tl.g);
                    ++issued;
                    if (++stage == stages) { stage = 0; phase ^= 1u; }
                }
            }
            if (lane == 0 && (!ok || *(volatile int *)&sh->abort_flag) && rank == 0) {
                // Drain: give the copies already issued a bounded chance to land before the CTA leaves.
                const int n = (int)(issued < stages ? issued : stages);
                int s2 = stage;
                uint32_t ph = phase;
                for (int i = 0; i < n; ++i) {
                    if (--s2 < 0) { s2 = stages - 1; ph ^= 1u; }
                    const uint32_t a = smem_u32(&sh->full[s2]);
                    const long long t0 = clock64();
                    while (!mbar_try_wait(a, ph) && clock64() - t0 < DRAIN_LIMIT_CYCLES) {}
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (rank 0 of the unit; whole warp, one elected lane issues) ------------------------------
        if (rank == 0) {
            constexpr uint32_t idesc0 = make_idesc(BL != kBTransposed, BC * CTAS);  // [E,K,N] and fractal are channel-contiguous
            const bool leader = elect_one();
            // descriptors of stage 0, MMA 0; the address field counts 16-byte units
            const uint32_t smem0 = smem_u32(smem);
            const uint64_t w_desc0 = weight_desc<SWIGLU && !DUAL, BL>(smem0);
            const uint64_t x_desc0 = make_smem_desc(smem0 + W_BYTES, 16, 1024, kSwizzle128);
            constexpr uint32_t W_STEP = weight_k_step(SWIGLU && !DUAL, BL) >> 4, X_STEP = UMMA_K >> 4;
            int stage = 0;
            uint32_t phase = 0;
            int buf = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            const uint32_t empty_peer = CTAS == 2 ? map_to_cta(&sh->empty[0], 1) : 0u;       // the partner's barriers
            const uint32_t acc_full_peer = CTAS == 2 ? map_to_cta(&sh->acc_full[0], 1) : 0u;
            int ti = 0;
            if (lane == 0) TRACE_GT(0, 0, 0);
            Tile next = unit < total_tiles ? decode_tile<MAX_TOK, BLOCK_GROUP>(sh, unit, p.n_tiles, L) : Tile{};
            for (int t = unit; t < total_tiles && ok; t += n_units, ++ti) {
                const Tile tl = next;
                if (tl.rows <= 0) break;
                const uint32_t idesc = idesc0 | (uint32_t)(((tl.rows + TOK_STEP - 1) / TOK_STEP * TOK_STEP) >> 3) << 17;
                if (lane == 0) TRACE(1, ti, 0);
                if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_empty[buf], acc_phase ^ 1u, sh, p.status, 200 + buf))) { ok = false; break; }
                if (lane == 0) TRACE(1, ti, 1);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)buf * BT;
                for (int kb = 0; kb < p.num_k_blocks; ++kb) {
#ifdef GMM_TRACE
                    const long long tw0 = clock64();
#endif
                    if (!__all_sync(0xffffffffu, mbar_wait<NZ && CTAS == 2>(&sh->full[stage], phase, sh, p.status, 300 + stage))) { ok = false; break; }
#ifdef GMM_TRACE
                    if (lane == 0) {
                        TRACE_ADD(1, ti, 3, clock64() - tw0);
                        TRACE_ADD(1, ti, 4, kb == 0 ? clock64() - tw0 : 0);
                    }
#endif
                    if (NZ) fence_async_proxy();
                    tc_fence_after();
                    if (leader) {
                        const uint64_t w_desc = w_desc0 + (uint64_t)(stage * (stage_bytes >> 4));
                        const uint64_t x_desc = x_desc0 + (uint64_t)(stage * (stage_bytes >> 4));
#pragma unroll
                        for (int j = 0; j < BK / UMMA_K; ++j) {
                            if (CTAS == 1) umma_i8(d_tmem, w_desc + j * W_STEP, x_desc + j * X_STEP, idesc, (kb | j) != 0 ? 1u : 0u);
                            if (DUAL) umma_i8(d_tmem + MAX_TOK, w_desc + (W_STAGE >> 4) + j * W_STEP, x_desc + j * X_STEP, idesc, (kb | j) != 0 ? 1u : 0u);
                            if (CTAS == 2) umma_i8_pair(d_tmem, w_desc + j * W_STEP, x_desc + j * X_STEP, idesc, (kb | j) != 0 ? 1u : 0u);
                        }
                        if (CTAS == 1) {
                            umma_commit(&sh->empty[stage]);
                        } else {  // the stage is free in both CTAs once these MMAs have read it
                            umma_commit_pair(smem_u32(&sh->empty[stage]));
                            umma_commit_pair(empty_peer + (uint32_t)stage * 8u);
                        }
                        if (kb == p.num_k_blocks - 1) {  // the tile's accumulators are complete
                            if (CTAS == 1) {
                                umma_commit(&sh->acc_full[buf]);
                            } else {
                                umma_commit_pair(smem_u32(&sh->acc_full[buf]));
                                umma_commit_pair(acc_full_peer + (uint32_t)buf * 8u);
                            }
                        }
                    }
                    __syncwarp();
                    if (kb == 0 && t + n_units < total_tiles) next = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t + n_units, p.n_tiles, L, tl.g);
                    if (++stage == stages) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (lane == 0) TRACE(1, ti, 2);
                if (lane == 0) TRACE_GT(0, 0, 1);
                buf ^= 1;
                if (buf == 0) acc_phase ^= 1u;
            }
        }
        else if (NZ) {
            // ------------------------------ rank 1, loader warps: token rows, and word to rank 0 that the stage is there ------------------------------
            // The loaders' weights are complete at this CTA's barrier; rank 0, which issues the MMA that reads them, has to learn
            // of it.  The chain, every link a rule of the PTX memory model: the loaders' cp.async are tracked by this CTA's
            // barrier (cp.async.mbarrier.arrive), whose completed phase this warp acquires; a proxy fence on that path orders
            // them before reads of the async proxy; a release at cluster scope, cumulative over what this warp has observed, with
            // the arrival at rank 0's barrier; rank 0's acquire at cluster scope, after which it issues the MMA.  The release
            // covers shared memory alone (sync_restrict): an arrival with an unrestricted one also waits for global memory, 1450
            // cycles per K block of 512.  The completion of the token copy would not do: it releases the copy's own bytes only.
            const bool leader = elect_one();
            const uint32_t full_rank0 = map_to_cta(&sh->full[0], 0);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int g_prev = 0;
            for (int t = unit; t < total_tiles && ok; t += n_units) {
                const Tile tl = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t, p.n_tiles, L, g_prev);
                if (tl.rows <= 0) break;
                g_prev = tl.g;
                const int my_tok = (tl.rows + TOK_STEP - 1) / TOK_STEP * TOK_STEP / CTAS;
                const int x_rows = x_box_rows<CTAS>(my_tok);
                const CUtensorMap *map_x = &maps_x.box[x_rows >= 128 ? 2 : x_rows >= 64 ? 1 : 0];
                const int kb_end = p.num_k_blocks - (t + n_units >= total_tiles ? p.skip_k_blocks : 0);
                for (int kb = 0; kb < kb_end; ++kb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&sh->full[stage], phase, sh, p.status, 330 + stage))) { ok = false; break; }
                    fence_async_proxy();
                    fence_release_shared_cluster();
                    if (leader) {
                        tma_load_2d<CTAS>(smem + stage * stage_bytes + W_BYTES, map_x, kb * BK, tl.row0 + my_tok, full_rank0 + (uint32_t)stage * 8u);
                        mbar_arrive_cluster_relaxed(full_rank0 + (uint32_t)stage * 8u);
                    }
                    __syncwarp();
                    if (++stage == stages) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (NZ && warp >= LD0) {
        // ------------------------------ weight loaders (FRACTAL_NZ) ------------------------------
        // Storage [E, N/32, K/16, 16, 32]: element (k, n) at (n/32 * K + k) * 32 + n%32.  A stage is 4 (two accumulators: 8) slabs
        // of 128 K-rows x 32 bytes; thread l takes 16-byte pieces l, l + 64, ... of each.  In shared memory a slab keeps that
        // order, except that the 16-byte halves of rows 4..7 of every 8 change places (32-byte swizzle).
        const int l = (int)threadIdx.x - LD0 * 32;
        const uint32_t dst0 = smem_u32(smem) + (uint32_t)((l * 16) ^ ((l * 2) & 16));
        constexpr int SLABS = W_BYTES / 4096;
        const size_t slab_bytes = (size_t)p.K * 32;
        const int8_t *w = static_cast<const int8_t *>(p.w_nz);
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        int g_prev = 0;
        for (int t = unit; t < total_tiles && ok; t += n_units) {
            const Tile tl = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t, p.n_tiles, L, g_prev);
            if (tl.rows <= 0) break;
            g_prev = tl.g;
            const int c0 = (tl.n_idx * CTAS + (int)rank) * CH_CTA, cols = SWIGLU ? p.half_n : p.N;
            const int8_t *src = w + (size_t)tl.g * p.K * p.N + (size_t)(c0 >> 5) * slab_bytes + l * 16;
            const size_t half_off = SWIGLU ? (size_t)(p.half_n >> 5) * slab_bytes : 0;   // from the activated to the linear half
            for (int kb = 0; kb < p.num_k_blocks; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&sh->empty[stage], phase ^ 1u, sh, p.status, 140 + stage))) { ok = false; break; }
                const uint32_t dst = dst0 + (uint32_t)(stage * stage_bytes);
                const int k_left = p.K - kb * BK - (l >> 1);   // > 0: this thread's K-row of the first piece exists
#pragma unroll
                for (int sl = 0; sl < SLABS; ++sl) {
                    constexpr int PER_HALF = SWIGLU ? SLABS / 2 : SLABS;
                    const int in_half = sl % PER_HALF;
                    const bool in_n = c0 + in_half * 32 < cols;
                    const int8_t *sp = src + (sl >= PER_HALF ? half_off : 0) + (size_t)in_half * slab_bytes;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool in = in_n && k_left > i * 32;
                        cp_async16(dst + (uint32_t)(sl * 4096 + i * 1024), in ? sp + i * 1024 : w, in ? 16u : 0u);
                    }
                }
                cp_async_arrive(&sh->full[stage]);
                src += BK * 32;
                if (++stage == stages) { stage = 0; phase ^= 1u; }
            }
        }
        cp_async_wait_all();
    } else if (warp < 2 + EPI_WARPS) {
        // ------------------------------ epilogue: warp -> (TMEM lane quarter, every second chunk of 32 tokens) ------------------------------
        const int quarter = warp & 3;
        const int chalf = (warp - 2) >> 2;
        const int te = (int)threadIdx.x - 64;  // the token whose factors this thread fetches (below BT)
        uint8_t *my_stage = sh->out_stage + (warp - 2) * WARP_STAGE_BYTES;
        uint8_t *half_stage = sh->out_stage + chalf * (CHUNK * ROW16_PITCH);
        constexpr int CHUNK_STEP = CHUNK * EPI_WARPS / 4;   // tokens from one of a warp's chunks to its next
        // swiglu: the warp of the other half (gate / up) with the same columns and tokens, two lane quarters on; the two share a
        // barrier
        const bool up = !DUAL && quarter >= 2;
        const int ch0 = SWIGLU && !DUAL ? (quarter & 1) * 32 : quarter * 32;   // first of this warp's 32 columns
        uint8_t *partner_stage = sh->out_stage + (chalf * 4 + ((quarter ^ 2) + 2) % 4) * WARP_STAGE_BYTES;
        uint64_t *grp_bar = &sh->grp_sync[SWIGLU ? chalf * 2 + (quarter & 1) : chalf];
        uint32_t grp_phase = 0;
        int buf = 0, it = 0;
        uint32_t acc_phase = 0;
        const uint64_t pol_last = policy_evict_last();
        bool ok = true;
        int g_prev = 0;
        for (int t = unit; t < total_tiles; t += n_units, ++it) {
            const Tile tl = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t, p.n_tiles, L, g_prev);
            if (tl.rows <= 0) break;
            g_prev = tl.g;
            const size_t sbase = (size_t)tl.g * p.N;
            const int c0 = (tl.n_idx * CTAS + (int)rank) * CH_CTA;   // first result column of this CTA

            // Per-channel values of this lane, and the factors of token te: all loads overlap the wait for the MMAs.
            constexpr int NCH = OUT16 ? 4 : 1;   // fragment rows lane/4 + 8j, else the lane's own channel
            float wsc[NCH], wsc_up = 0.0f;       // wsc_up: the linear half's, where the lane holds both
            float bias_f[NCH];
            int bias_i[NCH];
            if (MODE != kModeInt32 || !PLAIN) {
#pragma unroll
                for (int j = 0; j < NCH; ++j) {
                    const int lc = OUT16 ? quarter * 32 + (lane >> 2) + 8 * j : ch0 + lane;
                    const int c = c0 + lc;
                    const bool in = c < (SWIGLU ? p.half_n : p.N);
                    const size_t col = sbase + (size_t)(SWIGLU && up ? p.half_n + c : c);
                    wsc[j] = MODE != kModeInt32 && in ? load_scale1(p.w_scale, p.w_scale_dtype, col) : 0.0f;
                    if (DUAL && in) wsc_up = load_scale1(p.w_scale, p.w_scale_dtype, col + p.half_n);
                    bias_f[j] = 0.0f;
                    bias_i[j] = 0;
                    if ((!PLAIN || COMBINE) && in) {
                        if (p.bias_dtype == kBF16) bias_f[j] = __uint_as_float((uint32_t)__ldg(reinterpret_cast<const uint16_t *>(p.bias) + col) << 16);
                        else if (!COMBINE && p.bias_dtype == kI32) bias_i[j] = __ldg(reinterpret_cast<const int *>(p.bias) + col);
                    }
                }
            }
            float xs = te < tl.rows ? 1.0f : 0.0f, lg = 1.0f;   // 0: rows of other groups, never stored, stay small
            if (te < tl.rows) {
                if (MODE != kModeInt32 && p.x_scale) xs = __ldg(p.x_scale + tl.row0 + te);
                if (COMBINE && p.logit) lg = __ldg(p.logit + tl.row0 + te);
            }
            // Where the rows go.  A lane looks up one token of a chunk (of 16-bit results the eight that its warp stores, else
            // all 32), loads its index a chunk ahead - the first one here, while the MMAs run - and settles the address once; the
            // lanes that store a row get it by a shuffle.  With four indices loaded and tested by every lane inside the chunk,
            // scattered rows cost the call a third (K=1024 N=2048, 32 groups of 1000 rows, us: plain 70, scattered 95, now 82).
            const int my_tk = OUT16 ? quarter * (CHUNK / 4) + (lane & (CHUNK / 4 - 1)) : lane;
            auto load_dest = [&](int tk) -> long long {   // row of the result, -1 for no token
                if (tk >= tl.rows) return -1;
                if (COMBINE) return p.row_index_i32 ? (long long)__ldg(reinterpret_cast<const int *>(p.row_index) + tl.row0 + tk)
                                                    : __ldg(reinterpret_cast<const long long *>(p.row_index) + tl.row0 + tk);
                return p.out_row_index ? __ldg(p.out_row_index + tl.row0 + tk) : (long long)(tl.row0 + tk);
            };
            long long next_dest = SCATTER ? load_dest(chalf * CHUNK + my_tk) : 0;
            if (te == 0) TRACE(2, it, 0);
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_full[buf], acc_phase, sh, p.status, 400 + buf))) { ok = false; break; }
            if (te == 0) TRACE(2, it, 1);
            if (COMBINE && it == 0) wait_for_init();
            tc_fence_after();
            if (MODE != kModeInt32) {
                if (EPI_THREADS == BT || te < BT) {
                    sh->tok_scale[buf][te] = COMBINE && p.logit ? (p.x_scale ? __fmul_rn(xs, lg) : lg) : xs;
                    if (COMBINE) sh->tok_logit[buf][te] = lg;
                }
                mbar_arrive(&sh->tok_ready[buf]);
                if (!__all_sync(0xffffffffu, mbar_wait(&sh->tok_ready[buf], acc_phase, sh, p.status, 500 + buf))) { ok = false; break; }
            }
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * BT;
            const float *tok = sh->tok_scale[buf];

            // 16 tokens of S, one column per lane: a token's 32 values are one line of the staging buffer, stored straight from
            // the registers; the row maxima (NaN left out, as fmaxf does) are reduced on their bits.  Through a transpose in shared
            // memory, whose accesses come out of the MMAs' operand bandwidth (64 of its 128 bytes per cycle are read, 64 written
            // by the copies), K=1024 N=2048 took 136 us instead of 118 with 64 groups of 400 rows, 20.3 / 18.5 with 4 of 64.
            auto store_s = [&](const float (&v)[16], int t0) {
                const int col = c0 + ch0 + lane;
                const bool in = col < p.half_n;
                float *dst = reinterpret_cast<float *>(p.out) + (size_t)(tl.row0 + t0) * p.half_n + col;
                uint32_t amax = 0;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float val = v[i];
                    if (in && t0 + i < tl.rows) st_global_hint(dst, val, pol_last);
                    dst += p.half_n;
                    const uint32_t m = __reduce_max_sync(0xffffffffu, in ? __float_as_uint(fmaxf(fabsf(val), 0.0f)) : 0u);
                    if (lane == i) amax = m;
                }
                if (lane < 16 && t0 + lane < tl.rows) atomicMax(p.amax_bits + tl.row0 + t0 + lane, amax);
            };
            if (DUAL) {
                for (int tc = chalf * 16; tc < tl.rows; tc += 32) {
                    uint32_t va[16], vb[16];
                    tmem_ld16(taddr + tc, va);
                    tmem_ld16(taddr + MAX_TOK + tc, vb);
                    tmem_ld_wait();
                    // (acc * x_scale) * w_scale
                    float act[16], gate[16];
                    dequant16(va, tok + tc, wsc[0], act);
                    dequant16(vb, tok + tc, wsc_up, gate);
                    swiglu16(act, gate);
                    store_s(act, tc);
                }
            }
            for (int tc = chalf * CHUNK; !DUAL && tc < tl.rows && ok; tc += CHUNK_STEP) {
                if (SWIGLU) {
                    // The gate warp finishes tokens 0..15 of the chunk, the up warp 16..31: each sends the other its values of
                    // the other's tokens.
                    const int own0 = tc + (up ? 16 : 0), other0 = tc + (up ? 0 : 16);
                    uint32_t va[16], vb[16];
                    tmem_ld16(taddr + other0, vb);
                    tmem_ld16(taddr + own0, va);
                    tmem_ld_wait();
                    float mine[16], theirs[16];   // (acc * x_scale) * w_scale
                    dequant16(vb, tok + other0, wsc[0], theirs);
#pragma unroll
                    for (int i = 0; i < 16; ++i) *reinterpret_cast<float *>(partner_stage + i * 128 + lane * 4) = theirs[i];
                    dequant16(va, tok + own0, wsc[0], mine);
                    if (!group_sync(grp_bar, grp_phase, sh, p.status, lane, 700)) { ok = false; break; }
                    float act[16], gate[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float other = *reinterpret_cast<const float *>(my_stage + i * 128 + lane * 4);
                        act[i] = up ? other : mine[i];
                        gate[i] = up ? mine[i] : other;
                    }
                    swiglu16(act, gate);
                    store_s(act, own0);
                    // the partner may write the next chunk's values here
                    if (!group_sync(grp_bar, grp_phase, sh, p.status, lane, 710)) { ok = false; break; }
                } else if (!OUT16) {
                    // 32-bit results: int32 accumulators, or the combine
                    //   t = float(acc) * scale[n]; t *= (per_token[m] * logit[m]); t += logit[m] * float(bias[n]);
                    //   y[row_index[m], n] += t  (ComputeDequantAndActivate, DataCopyPerTokenScaleAndBrcb, VectorAtomicProcess
                    //   of gmm/grouped_matmul_finalize_routing/op_kernel/grouped_matmul_finalize_routing.h:418-448, 497-545, 343-366)
                    uint32_t v[32];
                    tmem_ld32(taddr + tc, v);
                    tmem_ld_wait();
                    // Four channels of a token per lane: L2 does an addition of four in the time of one (combine, K=2048 N=7168, 4096
                    // tokens x 8 over 32 experts: 504 us, 580 singly), and results that go to HBM are better off with four lines per
                    // store than with one straight from the registers (int32 of the same size 407 / 415; of K=1024 N=2048, 64 groups
                    // of 400 rows, 81 / 79.5).
                    const int col = c0 + quarter * 32 + (lane & 7) * 4;
                    uint32_t *const out = reinterpret_cast<uint32_t *>(p.out);   // rows of N 32-bit results
                    unsigned long long row_addr = 0;   // of token tc + lane; 0: not stored
                    if (SCATTER) {
                        const long long row = next_dest;
                        next_dest = load_dest(tc + CHUNK_STEP + lane);
                        if ((unsigned long long)row < p.row_limit) row_addr = reinterpret_cast<unsigned long long>(out + (size_t)row * p.N);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int t0 = tc + h * 16;
                        if (t0 >= tl.rows) break;
                        uint32_t r[16];
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            const int a0 = (int)v[h * 16 + i], a1 = (int)v[h * 16 + i + 1];
                            if (COMBINE) {
                                float2 t = unpair2(mul2(mul2(pair2(__int2float_rn(a0), __int2float_rn(a1)), pair2(wsc[0], wsc[0])),
                                                        *reinterpret_cast<const f32x2 *>(tok + t0 + i)));
                                if (p.bias_dtype == kBF16) {
                                    t.x = __fadd_rn(t.x, __fmul_rn(sh->tok_logit[buf][t0 + i], bias_f[0]));
                                    t.y = __fadd_rn(t.y, __fmul_rn(sh->tok_logit[buf][t0 + i + 1], bias_f[0]));
                                }
                                r[i] = __float_as_uint(t.x);
                                r[i + 1] = __float_as_uint(t.y);
                            } else {
                                r[i] = (uint32_t)(PLAIN ? a0 : a0 + bias_i[0]);
                                r[i + 1] = (uint32_t)(PLAIN ? a1 : a1 + bias_i[0]);
                            }
                        }
                        uint4 o[4];
                        transpose16(my_stage, r, lane, o);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int tk = h * 16 + i * 4 + (lane >> 3);   // of the chunk
                            uint32_t *row = SCATTER ? reinterpret_cast<uint32_t *>(__shfl_sync(0xffffffffu, row_addr, tk))
                                            : tc + tk < tl.rows ? out + (size_t)(tl.row0 + tc + tk) * p.N : nullptr;
                            if (!row || col >= p.N) continue;
                            if (COMBINE && p.scatter_add)
                                red_add_v4(reinterpret_cast<float *>(row + col), make_float4(__uint_as_float(o[i].x), __uint_as_float(o[i].y), __uint_as_float(o[i].z), __uint_as_float(o[i].w)));
                            else *reinterpret_cast<uint4 *>(row + col) = o[i];
                        }
                    }
                } else {
                    // 16-bit results.  After the exchange lane l of this warp stores 16 bytes (8 channels) of rows
                    // 2 i + l / 16 of its quarter of the chunk: a store instruction covers 256 contiguous bytes of two rows.
                    const int pc = lane & 15;
                    const int col = c0 + pc * 8;
                    constexpr int N8 = CHUNK / 8;   // 8-token pieces of the chunk
                    uint32_t v0[4 * N8], v1[4 * N8];
                    tmem_ld16x256b(taddr + tc, v0);
                    tmem_ld16x256b(taddr + (16u << 16) + tc, v1);
                    unsigned long long row_addr = 0;   // of token tc + my_tk; 0: not stored
                    if (SCATTER) {
                        long long row = next_dest, gpu_field = 0;
                        next_dest = load_dest(tc + CHUNK_STEP + my_tk);
                        uint16_t *obase = reinterpret_cast<uint16_t *>(p.out);
                        if (p.num_peers > 0) {  // high bits: which GPU's buffer, low 40 bits: row in it
                            gpu_field = row >> 40;
                            row &= (1ll << 40) - 1;
                            obase = reinterpret_cast<uint16_t *>(p.out_peers[gpu_field >= 0 && gpu_field < p.num_peers ? (int)gpu_field : 0]);
                        }
                        // an index that names no peer or no row of the result is skipped and reported, not stored
                        if (tc + my_tk < tl.rows) {
                            if ((unsigned long long)row < p.row_limit && (p.num_peers <= 0 || (unsigned long long)gpu_field < (unsigned long long)p.num_peers)) {
                                row_addr = reinterpret_cast<unsigned long long>(obase + (size_t)row * p.N);
                            } else if (lane < CHUNK / 4 && atomicCAS(p.status, kStatusOk, kStatusBadIndex) == kStatusOk) {
                                p.status[1] = (int)blockIdx.x;
                                p.status[2] = 800;
                                p.status[3] = tl.row0 + tc + my_tk;
                            }
                        }
                    }
                    tmem_ld_wait();
                    // Of every 8 tokens this lane holds two (4 i + its column pair) for four channels (lane / 4 + 8 j):
                    // (acc * w_scale) * x_scale, optional bias, optional activation, then one rounding
                    float o[N8][4][2];
#pragma unroll
                    for (int i = 0; i < N8; ++i) {
                        const f32x2 ts = *reinterpret_cast<const f32x2 *>(tok + tc + i * 8 + (lane & 3) * 2);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            int a0 = (int)(j < 2 ? v0[i * 4 + j * 2] : v1[i * 4 + (j - 2) * 2]);
                            int a1 = (int)(j < 2 ? v0[i * 4 + j * 2 + 1] : v1[i * 4 + (j - 2) * 2 + 1]);
                            if (!PLAIN) { a0 += bias_i[j]; a1 += bias_i[j]; }
                            f32x2 t = mul2(pair2(__int2float_rn(a0), __int2float_rn(a1)), pair2(wsc[j], wsc[j]));
                            if (PLAIN || p.x_scale) t = mul2(t, ts);
                            const float2 f = unpair2(t);
                            o[i][j][0] = f.x;
                            o[i][j][1] = f.y;
                        }
                    }
                    if (!PLAIN) {
                        if (p.bias_dtype == kBF16) {
#pragma unroll
                            for (int i = 0; i < N8; ++i)
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    o[i][j][0] = __fadd_rn(o[i][j][0], bias_f[j]);
                                    o[i][j][1] = __fadd_rn(o[i][j][1], bias_f[j]);
                                }
                        }
                        activate(p.act_type, reinterpret_cast<float(&)[8 * N8]>(o));
                    }
                    const bool f16 = EPI == kEpiHalf || EPI == kEpiHalfScatter || (!PLAIN && p.out_f16);
#pragma unroll
                    for (int i = 0; i < N8; ++i) {
                        uint32_t pk[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) pk[j] = f16 ? pack_f16x2(o[i][j][0], o[i][j][1]) : pack_bf16x2(o[i][j][0], o[i][j][1]);
                        stmatrix_x4_trans(smem_u32(half_stage + (i * 8 + (lane & 7)) * ROW16_PITCH + quarter * 64 + (lane >> 3) * 16),
                                          pk[0], pk[1], pk[2], pk[3]);
                    }
                    if (!group_sync(grp_bar, grp_phase, sh, p.status, lane, 720)) { ok = false; break; }
#pragma unroll
                    for (int i = 0; i < N8; ++i) {
                        const int r = quarter * (CHUNK / 4) + i * 2 + (lane >> 4);
                        const uint4 val = *reinterpret_cast<const uint4 *>(half_stage + r * ROW16_PITCH + pc * 16);
                        if (SCATTER) {
                            uint16_t *row = reinterpret_cast<uint16_t *>(__shfl_sync(0xffffffffu, row_addr, i * 2 + (lane >> 4)));
                            if (row && col < p.N) *reinterpret_cast<uint4 *>(row + col) = val;
                        } else if (tc + r < tl.rows && col < p.N) {
                            *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(p.out) + (size_t)(tl.row0 + tc + r) * p.N + col) = val;
                        }
                    }
                    // the other warps may write the next chunk's values
                    if (!group_sync(grp_bar, grp_phase, sh, p.status, lane, 730)) { ok = false; break; }
                }
            }
            if (!ok) break;
            if (te == 0) TRACE(2, it, 2);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->acc_empty[buf]);  // the buffer may be overwritten once every epilogue warp of the unit has read it
            buf ^= 1;
            if (buf == 0) acc_phase ^= 1u;

            if (SWIGLU) {
                // Tell the publishing lane that this warp's part of the tile is stored.  A CTA-wide release is enough here: the
                // lane's own fence is cumulative over what it has observed, so only one thread waits for the stores to reach
                // L2 (with a device-wide fence in every epilogue thread the warps stood still for 5000 cycles per tile).
                if (lane == 0) {
                    __threadfence_block();
                    atomicAdd(&sh->stored_count, 1u);
                }
                if (te == 0) TRACE(2, it, 3);
            }
        }
        if (SCATTER && p.num_peers > 0) __threadfence_system();  // rows stored into other GPUs' memory
        if (SWIGLU && ok) {  // nothing left to multiply: the last list is worked off by these warps, too
            const bool got = list_wait(&sh->wk_closing, 0u, sh, p.status, 660, 2ll * p.pace_cycles);
            if (__all_sync(0xffffffffu, got)) work_off(p, sh, sh->closing_slot, RQ + warp - 2, RQ + EPI_WARPS);
        }
    }

    else if (SWIGLU && warp > 2 + EPI_WARPS) {
        // ------------------------------ requantising warps (swiglu_quant) ------------------------------
        // A list names row blocks of which this unit has done tiles and which are complete by then; their rows are read while they
        // are still in L2.  With block_group row blocks at a time it is normally those of the unit's previous tiles, one after the
        // other as their last channel tile is done.  These warps spend their time waiting for L2; beside the epilogue that costs
        // nothing, inside it every tile of a C2-sized launch lost 13 of 36 thousand cycles to it, more than its MMAs take.
        const int w = warp - 3 - EPI_WARPS;
        for (int list = 0;; ++list) {
            const int ws = list % WK_DEPTH;
            const bool got = list_wait(&sh->wk_full[ws], ((uint32_t)(list / WK_DEPTH)) & 1u, sh, p.status, 650 + ws, 2ll * p.pace_cycles);
            if (!__all_sync(0xffffffffu, got)) break;
            const bool last = sh->work_last[ws] != 0;
            work_off(p, sh, ws, w, last ? RQ + EPI_WARPS : RQ);
            if (last) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->wk_empty[ws]);
        }
    }

    else if (SWIGLU) {
        // ------------------------------ publishing lane (swiglu_quant) ------------------------------
        // Per tile of this unit, in the epilogue's order: wait until every epilogue warp has stored the tile, arrive at its
        // row block, collect the row slices that fall to this CTA now (publish_and_collect) into the next work list, and pass
        // the list on if there is anything in it.  The last list takes or hands over what is still pending as well.  Nothing
        // here waits for another CTA; the only back-pressure is the ring of work lists, which the requantising warps empty.
        if (lane == 0) {
            int it = 0, list = 0, ws = 0;
            bool ok = true;
            int g_prev = 0;
            sh->n_work[0] = 0;
            auto pass_on = [&](bool last) {
                sh->work_last[ws] = last ? 1 : 0;
                if (last) sh->closing_slot = ws;
                __threadfence();
                mbar_arrive(&sh->wk_full[ws]);
                if (last) {
                    mbar_arrive(&sh->wk_closing);
                    return;
                }
                ++list;
                ws = list % WK_DEPTH;
                ok = mbar_wait(&sh->wk_empty[ws], (((uint32_t)(list / WK_DEPTH)) & 1u) ^ 1u, sh, p.status, 630 + ws);
                if (ok) sh->n_work[ws] = 0;
            };
            for (int t = unit; t < total_tiles && ok; t += n_units, ++it) {
                const Tile tl = decode_tile<MAX_TOK, BLOCK_GROUP>(sh, t, p.n_tiles, L, g_prev);
                if (tl.rows <= 0) break;
                g_prev = tl.g;
                // A block with tiles in the last wave that are cut into pieces counts in pieces: a whole tile has the shares of
                // its pieces, a piece one.
                PendingBlock mine;
                mine.rb = tl.block;
                mine.row0 = tl.block_row0;
                mine.rows = tl.block_rows;
                int pieces = 1;
                if (tl.block_last >= sh->split_from) {
                    const int sub = piece_tokens(tl.block_rows, sh->split);
                    pieces = (tl.block_rows + sub - 1) / sub;
                }
                mine.weight = tl.index < sh->split_from ? pieces : 1;
                mine.shares = p.n_tiles * CTAS * pieces;
                const unsigned need = (unsigned)(it + 1) * EPI_WARPS;
                if (*(volatile unsigned *)&sh->stored_count < need) {
                    const long long t0 = clock64();
                    while (*(volatile unsigned *)&sh->stored_count < need) {
                        __nanosleep(60);
                        if (*(volatile int *)&sh->abort_flag) { ok = false; break; }
                        if (clock64() - t0 > sh->wait_limit) {
                            *(volatile int *)&sh->abort_flag = 1;
                            if (atomicCAS(p.status, kStatusOk, kStatusWaitTimeout) == kStatusOk) {
                                p.status[1] = (int)blockIdx.x;
                                p.status[2] = 620;
                                p.status[3] = it;
                            }
                            ok = false;
                            break;
                        }
                    }
                    if (!ok) break;
                }
                TRACE(3, it, 0);
                __threadfence();
                if (mine.rb < p.max_blocks) publish_and_collect(p, sh, ws, mine);   // beyond: a list that is reported (build_schedule)
                TRACE(3, it, 2);
                TRACE_ADD(3, it, 3, sh->n_work[ws]);
                if (sh->n_work[ws] > 0) pass_on(false);
                *(volatile unsigned *)&sh->published = (unsigned)it + 1;
            }
            if (ok && !*(volatile int *)&sh->abort_flag) {
                release_pending(p, sh, ws, 2ll * p.pace_cycles);
                pass_on(true);
            }
        }
    }

    if (COMBINE && warp == 0) wait_for_init();
    __syncthreads();
    if (CTAS == 2) cluster_sync_all();  // neither CTA leaves, or frees TMEM, while the other can still reach into it
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc<CTAS>(tmem_base, TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

template <int MODE, int BL, int EPI, int CTAS>
cudaError_t launch_variant(const Plan &plan, const KParams &kp, cudaStream_t stream)
{
    auto kern = gmm_w8a8_sm100_kernel<MODE, BL, EPI, CTAS>;
    // Once per device and instantiation; the attribute is idempotent, so a race only repeats the call.
    static unsigned long long done_mask = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!((done_mask >> (dev & 63)) & 1ull)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
        if (e != cudaSuccess) return e;
        done_mask |= 1ull << (dev & 63);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CTAS == 2 ? (plan.num_sms & ~1) : plan.num_sms), 1, 1);
    cfg.blockDim = dim3(num_threads(MODE, BL, EPI), 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (CTAS == 2) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs].val.clusterDim.x = CTAS;
        attr[attrs].val.clusterDim.y = 1;
        attr[attrs++].val.clusterDim.z = 1;
    }
    if (EPI == kEpiCombine && plan.beside_init) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    XMaps maps_x;
    for (int i = 0; i < X_MAPS; ++i) maps_x.box[i] = plan.map_x[i];
    cfg.attrs = attr;
    cfg.numAttrs = (unsigned)attrs;
    return cudaLaunchKernelEx(&cfg, kern, maps_x, plan.map_w, kp);
}

template <int MODE, int BL, int EPI>
cudaError_t launch_ctas(const Plan &plan, const KParams &kp, cudaStream_t stream)
{
    return plan.ctas == 2 ? launch_variant<MODE, BL, EPI, 2>(plan, kp, stream) : launch_variant<MODE, BL, EPI, 1>(plan, kp, stream);
}

template <int MODE, int BL>
cudaError_t launch_epi(int epi, const Plan &plan, const KParams &kp, cudaStream_t stream)
{
    if (MODE == kModeSwigluQuant || epi == kEpiPlain) return launch_ctas<MODE, BL, kEpiPlain>(plan, kp, stream);
    if (epi == kEpiScatter) return launch_ctas<MODE, BL, kEpiScatter>(plan, kp, stream);
    if (MODE == kModeDequantBf16 && epi == kEpiHalf) return launch_ctas<MODE, BL, MODE == kModeDequantBf16 ? kEpiHalf : kEpiPlain>(plan, kp, stream);
    if (MODE == kModeDequantBf16 && epi == kEpiHalfScatter) return launch_ctas<MODE, BL, MODE == kModeDequantBf16 ? kEpiHalfScatter : kEpiPlain>(plan, kp, stream);
    if (MODE == kModeDequantBf16 && epi == kEpiCombine) return launch_ctas<MODE, BL, MODE == kModeDequantBf16 ? kEpiCombine : kEpiPlain>(plan, kp, stream);
    return launch_ctas<MODE, BL, kEpiGeneric>(plan, kp, stream);
}

template <int MODE>
cudaError_t launch_layout(int layout, int epi, const Plan &plan, const KParams &kp, cudaStream_t stream)
{
    if (layout == kBTransposed) return launch_epi<MODE, kBTransposed>(epi, plan, kp, stream);
    if (layout == kBFractalNz) return launch_epi<MODE, kBFractalNz>(epi, plan, kp, stream);
    return launch_epi<MODE, kBRowMajor>(epi, plan, kp, stream);
}

}  // namespace

// The tcgen05 path needs 16-byte aligned row pitches for TMA (K for x; N or K for the weight), 16-byte
// aligned base pointers and, for SwiGLU, a half width that keeps the second box aligned.
bool sm100_shape_ok(const Problem &p)
{
    if (p.K % 16 != 0 || p.N % 16 != 0) return false;
    if (p.mode == kModeSwigluQuant && p.N % 32 != 0) return false;
    if (p.w_layout == kBFractalNz && (p.N % 32 != 0 || (p.mode == kModeSwigluQuant && p.N % 64 != 0))) return false;
    if (p.gl_len > MAX_GROUPS || p.gl_len <= 0) return false;
    if (p.M <= 0 || p.M > 0x7fffffffll / 2 || p.K > 0x7fffffffll || p.N > 0x7fffffffll) return false;
    if ((reinterpret_cast<uintptr_t>(p.x) & 15) || (reinterpret_cast<uintptr_t>(p.w) & 15)) return false;
    if (reinterpret_cast<uintptr_t>(p.out0) & 15) return false;
    if (reinterpret_cast<uintptr_t>(p.w_scale) & 3) return false;
    if (p.bias && (reinterpret_cast<uintptr_t>(p.bias) & 3)) return false;
    if (p.mode == kModeSwigluQuant && (!p.out1 || (reinterpret_cast<uintptr_t>(p.out1) & 3))) return false;
    return true;
}

cudaError_t sm100_encode_maps(const Problem &p, Plan &plan)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    // x: boxes of 32, 64 and 128 rows, of which the producer takes the one that covers a tile's share
    for (int i = 0; i < X_MAPS; ++i) {
        cuuint64_t dims[2] = {(cuuint64_t)p.K, (cuuint64_t)p.M};
        cuuint64_t strides[1] = {(cuuint64_t)p.K};
        cuuint32_t box[2] = {BK, 32u << i};
        cuuint32_t estr[2] = {1, 1};
        CUresult r = enc(&plan.map_x[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(p.x), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    // weights: a box is 128 channels x 128 K; with swiglu_quant 64 (pair) or 128 channels of either half of the
    // columns, the halves being a dimension of their own
    const cuuint32_t halves = p.mode == kModeSwigluQuant ? 2 : 1, box_ch = halves == 2 && plan.ctas == 2 ? BC / 2 : BC;
    const cuuint64_t K = (cuuint64_t)p.K, N = (cuuint64_t)p.N, cols = N / halves, E = (cuuint64_t)p.E;
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r;
    if (p.w_layout == kBFractalNz) {
        plan.map_w = plan.map_x[0];  // the loader warps read it; the kernel's map parameter is not used
        return cudaSuccess;
    }
    if (p.w_layout == kBTransposed) {  // [E, N, K]
        cuuint64_t dims[4] = {K, cols, halves, E};
        cuuint64_t strides[3] = {K, K * cols, K * N};
        cuuint32_t box[4] = {BK, box_ch, halves, 1};
        r = enc(&plan.map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t *>(p.w), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {  // [E, K, N]
        cuuint64_t dims[4] = {cols, K, halves, E};
        cuuint64_t strides[3] = {N, cols, K * N};
        cuuint32_t box[4] = {box_ch, BK, halves, 1};
        r = enc(&plan.map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t *>(p.w), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, box_ch == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    return cudaSuccess;
}

cudaError_t sm100_launch(const Problem &p, Plan &plan, void *workspace, cudaStream_t stream)
{
    plan.num_sms = device_sm_count();
    if (plan.num_sms <= 0) return cudaErrorNoDevice;
    if (p.opt.max_ctas > 0 && p.opt.max_ctas < plan.num_sms) plan.num_sms = p.opt.max_ctas;
    if (plan.ctas != 2 || plan.num_sms < 2) plan.ctas = 1;  // a CTA pair needs two CTAs
    cudaError_t e = sm100_encode_maps(p, plan);
    if (e != cudaSuccess) return e;
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    KParams kp;
    kp.group_list = p.group_list;
    kp.gl_len = p.gl_len;
    kp.gl_type = p.gl_type;
    kp.M = (int)p.M;
    kp.K = (int)p.K;
    kp.N = (int)p.N;
    kp.half_n = (int)(p.N / 2);
    const int64_t tile_cols = p.mode == kModeSwigluQuant ? BC : BC * plan.ctas, cols = p.mode == kModeSwigluQuant ? p.N / 2 : p.N;
    kp.n_tiles = (int)((cols + tile_cols - 1) / tile_cols);
    kp.max_blocks = plan.row_blocks < 0x7fffffffll ? (int)plan.row_blocks : 0x7fffffff;
    kp.max_tiles = p.mode == kModeSwigluQuant ? (int)(plan.row_blocks * kp.n_tiles < 0x7fffffffll ? plan.row_blocks * kp.n_tiles : 0x7fffffffll) : 0x7fffffff;
    kp.num_k_blocks = (int)((p.K + BK - 1) / BK);
    kp.w_nz = p.w;
    kp.w_scale = p.w_scale;
    kp.w_scale_dtype = p.w_scale_dtype;
    kp.x_scale = p.x_scale;
    kp.bias = p.bias;
    kp.bias_dtype = p.bias ? p.bias_dtype : kNone;
    kp.act_type = p.act_type;
    kp.out_f16 = p.out_f16;
    kp.status = reinterpret_cast<int *>(ws + plan.off_status);
    kp.amax_bits = reinterpret_cast<unsigned *>(ws + plan.off_amax);
    kp.rb_counter = reinterpret_cast<int *>(ws + plan.off_done);
    kp.out_row_index = reinterpret_cast<const long long *>(p.out_row_index);
    kp.q_out = reinterpret_cast<int8_t *>(p.out0);
    kp.q_scale_out = reinterpret_cast<float *>(p.out1);
    kp.out = p.mode == kModeSwigluQuant ? static_cast<void *>(ws + plan.off_stage) : p.out0;

    // The generic epilogue is for bias and activation alone: its sixteen warps only get in the way of the MMAs where a chunk's
    // arithmetic is short.  Without the tokens' scales the plain arithmetic multiplies by one; fp16 rows have instances of their own.
    // K=2048 N=7168, 32 groups of 1024 rows, us with the generic epilogue on eight warps / on sixteen / now: fp16 369 / 379 / 340, scattered
    // 371 / 381 / 353; bf16 without the tokens' scales 354 / 363 / 326 (bf16 with them 323).
    const int epi = p.combine ? kEpiCombine : p.bias || p.act_type ? kEpiGeneric
                  : p.out_f16 ? (p.out_row_index ? kEpiHalfScatter : kEpiHalf) : (p.out_row_index ? kEpiScatter : kEpiPlain);
    kp.logit = p.logit;
    kp.row_index = p.row_index;
    kp.row_index_i32 = p.row_index_i32;
    kp.scatter_add = p.scatter_add;
    kp.row_limit = p.combine || p.out_rows > 0 ? (unsigned long long)p.out_rows : 1ull << 62;
    if (p.combine && (p.mode != kModeDequantBf16 || !p.row_index)) return cudaErrorInvalidValue;
    kp.num_peers = p.mode == kModeDequantBf16 ? p.num_peers : 0;
    for (int i = 0; i < 8; ++i) kp.out_peers[i] = i < kp.num_peers ? p.out_peers[i] : nullptr;
    if (kp.num_peers > 0 && (epi != kEpiScatter || !p.x_scale)) return cudaErrorInvalidValue;
    // Pacing (see the producer): needs one zeroed word per wave; the plan reserves them only where it pays.
    // The plan reserves a counter per tile, so there is one for every wave; a single unit has nobody to keep pace with.
    kp.wave_cnt = plan.off_wave && plan.num_sms >= 2 ? reinterpret_cast<int *>(ws + plan.off_wave) : nullptr;
    kp.pace_cycles = kp.num_k_blocks * 1200 + 20000;   // about one tile's duration
#ifdef GMM_TRACE
    kp.trace = getenv("GMM_TRACE_PTR") ? reinterpret_cast<long long *>(strtoull(getenv("GMM_TRACE_PTR"), nullptr, 0)) : nullptr;
#endif
    if (const char *e = getenv("GMM_B200_PACE")) {
        if (e[0] == '0') kp.wave_cnt = nullptr;
        else if (atoi(e) > 1) kp.pace_cycles = atoi(e);
    }
    kp.wait_limit = p.opt.wait_limit_cycles > 0 ? p.opt.wait_limit_cycles : WAIT_LIMIT_CYCLES;
    kp.skip_k_blocks = p.opt.test_skip_k_blocks > 0 ? (p.opt.test_skip_k_blocks < kp.num_k_blocks ? p.opt.test_skip_k_blocks : kp.num_k_blocks) : 0;
    if (p.opt.ev_start) cudaEventRecord(p.opt.ev_start, stream);
    if (p.mode == kModeSwigluQuant) e = launch_layout<kModeSwigluQuant>(p.w_layout, epi, plan, kp, stream);
    else if (p.mode == kModeInt32) e = launch_layout<kModeInt32>(p.w_layout, epi, plan, kp, stream);
    else e = launch_layout<kModeDequantBf16>(p.w_layout, epi, plan, kp, stream);
    if (p.opt.ev_stop) cudaEventRecord(p.opt.ev_stop, stream);
    return e;
}

}  // namespace gmm
