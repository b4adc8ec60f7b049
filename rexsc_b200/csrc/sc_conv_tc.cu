// SC conv forward on the 5th-generation tensor cores (tcgen05, 4-bit operands, fp32 accumulators in TMEM).
//
// Per time slot t the count that OR-n saturates is a plain contraction of 0/1 values,
//     count_t[pixel][sign, co] = sum_{tap, c} a_t[pixel + tap][c] * w_t[sign, co][tap, c],
// and only min(count_t, n) is non-linear -- it is applied to the finished accumulator of every slot:
//     out[pixel][sign, co] = sum_t min(count_t, n)            (sc_device.cu:127-151 of the reference).
// So every slot is one GEMM with M = 128 rows (64 output channels x {positive, negative} weight stream, the TMEM
// lanes), N = output-pixel candidates, K = taps x channels, issued as tcgen05.mma.kind::mxf4 M128 N160 K64.
//
// Why 4-bit floats.  0 and the powers of two that the operands use (0.5, 1, 2) are exact e2m1 numbers, every block
// scale is 1, a coincidence contributes exactly 1.0 and fp32 accumulators count exactly to 2^24.  One more MMA per unit
// and slot starts the accumulators at 2^23, so that the low 16 bits of each ARE the integer count and a packed TMEM read
// delivers two per register.  Against the int8 kind the same channels take half the operand bytes and half the MMA time, and
// expanding 32 bits into 32 operands takes 5 logic instructions instead of 17.
//
// Why the weights are the TMEM operand.  The MMA reads its M operand from tensor memory and its N operand from shared
// memory; with both in shared memory (128 x 128 tiles) operand reads alone fill the shared-memory pipe (8 KB per 64
// clk).  The pixels have to stay in shared memory, because a filter tap is the same buffer at another start row; the
// weights have no such need, are expanded straight from registers into TMEM columns, and leave 64 B/clk of operand
// reads.
//
// Columns.  The N dimension runs over the "origin grid": per image Ho x Wo candidates (i, j), candidate (i, j) being
// the padded-input pixel (i*stride_h, j*stride_w), i.e. the top-left tap of output pixel (i, j) when i < OH and
// j < OW (other candidates are computed and dropped; they are the padding of the grid, a few percent).  A tile is 320
// consecutive candidates, two MMA column blocks ("units") of 160.
//
// Operands are generated from bit planes (one bit per element and slot, 32 channels per word):
//   pixels   the slot's activation bits of the tile's patch as 16-byte K-columns [32-channel word][patch row][16 B]
//            (unswizzled K-major, rows 16 bytes apart).  The patch is kept as one plane per stride residue
//            (kh % stride_h, kw % stride_w); inside a plane, row r holds the pixel of that residue that belongs to
//            candidate o0 + r.  The operand of filter tap (kh, kw) is then the SAME buffer with its start address moved
//            to plane(kh % sh, kw % sw) + (kh / sh) * Wo + kw / sw rows: no im2col, for any stride.
//   weights  the slot's weight bits, TMEM columns [tap][32-channel word][4 columns of 8 nibbles].
//
// Tensor memory (512 columns): two accumulator units of 160, two operand buffers of up to 72, 2 x 16 columns of block
// scales (the same columns serve both operands), 8 of the bias MMA's weights.
//
// One persistent CTA per SM walks its tiles as a single pipeline (a tile's first loads and its store overlap the
// neighbouring tiles' MMAs): 16 warps fold counts, eight expand operands, one copies weight words, one issues the MMAs,
// unit 0 then unit 1 of every step.  A pipeline step is one slot x one chunk of 64 channels (1x1 filters: up to 256).  Operand buffers are
// double-buffered, a unit's accumulators are folded while the other unit is computed, and every dependence is an
// mbarrier phase: while the tensor core works through step i, the folding warps are on the unit that finished and
// the expanding warps write the operands of step i+1.
// Every wait is bounded; on a time-out the CTA reports through the status word, frees its TMEM and returns.
#include "common.cuh"
#include <stdlib.h>

namespace rexsc {

namespace {

constexpr int kTcFoldWarps = 16;            // warps that fold finished accumulators into running sums, eight per unit
constexpr int kTcExpandWarps = 8;           // warps that expand operands, two per TMEM lane quarter
constexpr int kTcIssueWarp = kTcFoldWarps + kTcExpandWarps; // issues the MMAs
constexpr int kTcLoadWarp = kTcIssueWarp + 1;               // copies the weight bit words into shared memory
constexpr int kTcThreads = (kTcFoldWarps + kTcExpandWarps + 4) * 32; // whole warpgroups: two warps idle
// Registers per thread: 896 threads are launched with 72, which the warpgroups share out again by what they need (the
// folding warps hold 40 sum and 40 count registers).
constexpr int kTcRegsLaunch = 72, kTcRegsFold = 96, kTcRegsExpand = 40, kTcRegsIssuer = 32;
static_assert(kTcFoldWarps * 32 * kTcRegsFold + kTcExpandWarps * 32 * kTcRegsExpand + 128 * kTcRegsIssuer <= kTcThreads * kTcRegsLaunch,
              "more registers than the block has");
constexpr int kTcMaxDepth = 4;              // pipeline steps whose bit words are in shared memory or on their way
constexpr int kTcBars = 9 + 2 * kTcMaxDepth;
constexpr int kTcUnit = 160;       // candidates of one MMA (its N)
constexpr int kTcM = 2 * kTcUnit;  // candidates per tile: two units that share one weight operand
constexpr int kTcCols = kTcUnit / 2; // accumulator columns of its unit that one warp folds
constexpr int kTcCout = 64;        // output channels per CTA
constexpr int kTcN = 2 * kTcCout;  // weight rows (MMA M, TMEM lanes): positive block [0,64), negative block [64,128)
constexpr int kTcMaxTaps = 9;      // filter taps whose weight operand is staged at once
constexpr int kTcMaxARows = 8;     // patch rows per expanding thread (all residue planes together)
// Which layers the path takes: residue planes x (256 + tap halo) up to this many rows.  The patch below would hold some
// more; but a layer on this path needs up to 14 times the workspace of the ALU kernels (bit planes of 32-channel words
// beside theirs, whichever kernel runs), so taking more layers would put calls that run today beyond the fixed scratch of
// rexsc_sc_conv2d_fwd_static, or beyond the card (stride 2 on 298 x 298 maps: 71 -> 165 GB at batch 691).
constexpr int kTcMaxPlaneRows = 1536, kTcPlaneTile = 256;
constexpr int kTcWordCols = 4;     // TMEM columns of one 32-channel weight word (8 nibbles per column)
constexpr int kTcMaxWords = 18;    // weight words per row and step: the operand buffers' TMEM columns / kTcWordCols
constexpr uint32_t kTcColA = 2 * kTcUnit;                                   // first column of the weight buffers
constexpr uint32_t kTcColSf = kTcColA + 2 * kTcMaxWords * kTcWordCols;      // block scales of the operands: 1
constexpr uint32_t kTcColSfBias = kTcColSf + 16;                            // block scales of the bias MMA: 2^11
constexpr uint32_t kTcColBias = kTcColSfBias + 16;                          // its weight operand: K element 0 is 2, the others 0
static_assert(kTcColBias + 8 <= 512, "tensor memory has 512 columns");
constexpr int kTcStageCols = 32;   // candidates that pass through a warp's store staging at a time
constexpr int kTcStagePitch = kTcStageCols / 2 + 1; // words per row of a warp's store staging: odd, so rows change banks
constexpr uint32_t kTcWaitLimit = 1u << 18; // try_wait attempts before a wait gives up (each may sleep kTcSuspendNs)
constexpr uint32_t kTcSuspendNs = 4000;    // a waiting warp sleeps in the barrier unit instead of spinning on issue slots

struct TcArgs {
    int OH, OW, KHW, Co, CW;
    int CK;          // pipeline steps per slot = ceil(CW / KWC)
    int depth;       // steps of bit words kept in shared memory: kTcMaxDepth, or 2 when it is short
    int nrh, nrw, Wq, Hrows, Wrow; // stored pixel grid (see tap_offset in common.cuh)
    int Ho, Wo;      // origin grid of one image
    int shift;       // candidates by which the patch starts BEFORE the tile's first candidate: 0, or Wo + 1 on the
                     // compact grid (ConvPlan::origin), whose candidates are the CENTRE taps of their output pixels
    int Mh;          // patch rows per residue plane: kTcM + largest in-plane tap shift, rounded up to 8
    int rows_a;      // patch rows of all planes
    int slots, n_or;
    long long total_o; // candidates = N * Ho * Wo
    int tiles_x;       // candidate tiles = ceil(total_o / kTcM)
    int total_tiles;   // tiles_x * (64-channel output chunks); tile index = chunk * tiles_x + x
    int out_al4;       // both output pointers are 4-byte aligned: two channels of a pixel may be stored at once
    int out_vec;       // ... 16-byte aligned, and so is every pixel's channel run: eight at once
    int balanced;      // 0: a CTA walks whole tiles blockIdx.x, + gridDim.x, ...
                       // 1: the (tile, time slot) pairs, in that order, are cut into gridDim.x equal runs, one per CTA.
                       //    A tile that two or more CTAs share is zeroed before the launch (zero_shared_tiles_kernel)
                       //    and every sharer adds its partial sums with packed 16-bit atomics; tiles that lie inside
                       //    one run are stored plainly.  No SM idles in a last, partly filled wave of tiles.
                       // 2: the same runs for outputs whose rows cannot take packed adds (NCHW, ragged or unaligned
                       //    channel runs): the host clears the whole outputs and every tile adds 16-bit values.
    long long NHWp;
    int out_nhwc;
    int tap_off[kTcMaxTaps]; // patch-row offset of every tap (kernel parameters are warp-uniform by construction)
};

// the tiles and time slots of CTA b of G (TcArgs::balanced)
struct TileRun {
    int first_tile, tile_stride, tiles; // tile k of the CTA = first_tile + k * tile_stride
    int slot_first;                     // first time slot of its first tile
    int slot_last_end;                  // end (exclusive) of the time slots of its last tile
    int slots;                          // time slots of all its tiles together
};

__host__ __device__ __forceinline__ TileRun tile_run(int total_tiles, int slots, int balanced, int b, int G)
{
    TileRun r;
    if (!balanced) {
        r.first_tile = b; r.tile_stride = G;
        r.tiles = (total_tiles - b + G - 1) / G;
        r.slot_first = 0; r.slot_last_end = slots;
        r.slots = r.tiles * slots;
    } else {
        // run b = units [u0, u1) of the total_tiles * slots (tile, slot) pairs; G <= units, so no run is empty
        const long long units = (long long)total_tiles * slots;
        const long long u0 = units * b / G, u1 = units * (b + 1) / G;
        const long long last = (u1 - 1) / slots;
        r.first_tile = (int)(u0 / slots); r.tile_stride = 1;
        r.tiles = (int)(last - r.first_tile) + 1;
        r.slot_first = (int)(u0 - (long long)r.first_tile * slots);
        r.slot_last_end = (int)(u1 - 1 - last * slots) + 1;
        r.slots = (int)(u1 - u0);
    }
    return r;
}

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// unswizzled K-major descriptor: rows 16 B apart (8-row core matrices back to back), K-columns `lbo_bytes` apart
__device__ __forceinline__ uint64_t desc_interleaved(uint32_t addr, uint32_t lbo_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3fff);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
    d |= (uint64_t)(128 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// (a polling loop of four instructions: waiting warps share issue slots with working ones)
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 left;\n\t"
        "mov.u32 left, %4;\n"
        "POLL_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "@p bra READY_%=;\n\t"
        "sub.u32 left, left, 1;\n\t"
        "setp.ne.u32 q, left, 0;\n\t"
        "@q bra POLL_%=;\n"
        "READY_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(kTcSuspendNs), "n"(kTcWaitLimit) : "memory");
    return ok != 0;
}

// 32 bits -> 32 e2m1 operands (16 bytes).  A bit expands by masking where it stands: bits 0, 1, 2 of a nibble are the
// numbers 0.5, 1 and 2, bit 3 (the sign) is moved down to 2 first.  The weight bit planes store every nibble
// bit-reversed, so that their numbers are 2, 1, 0.5 and 0.5: every coincidence contributes exactly 1.  Both operands
// thereby permute the channels of a word in the same way, which a sum does not notice.
__device__ __forceinline__ uint4 spread_pixels(uint32_t h)
{
    return make_uint4(h & 0x11111111u, h & 0x22222222u, h & 0x44444444u, (h >> 1) & 0x44444444u);
}
__device__ __forceinline__ uint4 spread_weights(uint32_t h)
{
    const uint32_t g = h >> 1;
    return make_uint4(g & 0x44444444u, g & 0x22222222u, g & 0x11111111u, h & 0x11111111u);
}

// 32 (16) TMEM columns as 16 (8) registers: the low 16 bits of two adjacent columns per register
#define REXSC_TMEM_LD32P(arr, taddr)                                                                                  \
    asm volatile(                                                                                                     \
        "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 "                                                           \
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"                              \
        : "=r"(arr[0]), "=r"(arr[1]), "=r"(arr[2]), "=r"(arr[3]), "=r"(arr[4]), "=r"(arr[5]), "=r"(arr[6]),           \
          "=r"(arr[7]), "=r"(arr[8]), "=r"(arr[9]), "=r"(arr[10]), "=r"(arr[11]), "=r"(arr[12]), "=r"(arr[13]),       \
          "=r"(arr[14]), "=r"(arr[15])                                                                                \
        : "r"(taddr)                                                                                                  \
        : "memory")
#define REXSC_TMEM_LD16P(arr, taddr)                                                                                  \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"            \
        : "=r"(arr[0]), "=r"(arr[1]), "=r"(arr[2]), "=r"(arr[3]), "=r"(arr[4]), "=r"(arr[5]), "=r"(arr[6]),           \
          "=r"(arr[7])                                                                                                \
        : "r"(taddr)                                                                                                  \
        : "memory")

// wait for the thread's TMEM reads; the registers are operands so that nothing that uses them can move ahead of it
#define REXSC_TMEM_WAIT16(arr)                                                                                        \
    asm volatile("tcgen05.wait::ld.sync.aligned;"                                                                     \
        : "+r"(arr[0]), "+r"(arr[1]), "+r"(arr[2]), "+r"(arr[3]), "+r"(arr[4]), "+r"(arr[5]), "+r"(arr[6]),           \
          "+r"(arr[7]), "+r"(arr[8]), "+r"(arr[9]), "+r"(arr[10]), "+r"(arr[11]), "+r"(arr[12]), "+r"(arr[13]),       \
          "+r"(arr[14]), "+r"(arr[15])                                                                                \
        :: "memory")
#define REXSC_TMEM_WAIT8(arr)                                                                                         \
    asm volatile("tcgen05.wait::ld.sync.aligned;"                                                                     \
        : "+r"(arr[0]), "+r"(arr[1]), "+r"(arr[2]), "+r"(arr[3]), "+r"(arr[4]), "+r"(arr[5]), "+r"(arr[6]),           \
          "+r"(arr[7])                                                                                                \
        :: "memory")

// KHW_T: taps known at compile time (9, 1) or 0 for any tap count up to kTcMaxTaps
// KWC:   32-channel words per pipeline step (even: one MMA takes two; above 4 only with KHW_T == 1)
// RA:    patch rows per expanding thread (1 .. kTcMaxARows)
//
// What bounds it, and the split of the warps.  The MMAs of a step take 18 x 83 clk on a 3x3 layer; everything else has
// to fit beside them, so the instruction count decides, and with it what every warp repeats per step: addresses, waits,
// hand-overs.  Measured on 64 -> 64 channels, 3x3, 56x56, 32 slots, batch 256 (accumulate launch alone; tensor pipe busy):
//   int8 operands, both in shared memory, 16 warps on both jobs            1.02 ms (80 % of an int8 pipe of half the rate)
//   4-bit, 16 such warps                                                    1.20 ms (43 %)
//   8 folding + 4 expanding warps                                           0.83 ms
//   16 folding (eight per unit) + 8 expanding, fp32 counts read in two goes 0.74 ms (59 %)
//   2^23 bias: packed counts, one read per unit and slot; 16-byte stores    0.64 ms
// of which the MMAs are 0.54 ms.  512 -> 512 channels, 7x7: 1.13 -> 0.60 ms, the MMAs alone.  1x1 filters on few channels
// stay bound by the hand-overs of a slot (MMA, commit, TMEM read, release: some 1600 clk for both units).
template <int KHW_T, int KWC, int RA>
__global__ void __launch_bounds__(kTcThreads, 1)
sc_conv_tc_kernel(TcArgs a, const uint32_t *__restrict__ Ab, const uint32_t *__restrict__ Wb,
                  int16_t *__restrict__ out_pos, int16_t *__restrict__ out_neg, int *__restrict__ status, int gate)
{
    static_assert(KWC % 2 == 0 && (KWC <= 4 || KHW_T == 1), "an MMA takes two words");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    // One of a pair of launches, of which the expand stage's verdict on the activation borders (status word 1: 0 =
    // the compact planes are valid) picks one: +1 runs on valid compact planes only, -1 on the standard planes that
    // replaced them.  The whole grid takes the same branch, before any barrier or tensor memory exists.
    if (gate != 0 && (gate > 0) == (status[1] != 0)) return;
    uint8_t *smem = smem_raw + ((128u - (saddr(smem_raw) & 127u)) & 127u);
    const int KHW = KHW_T ? KHW_T : a.KHW;
    const uint32_t a_bytes = (uint32_t)KWC * (uint32_t)a.rows_a * 16u; // [KWC words][rows_a][16]
    uint32_t *stage_all = reinterpret_cast<uint32_t *>(smem + 2 * a_bytes); // [fold warp][32 rows][kTcStagePitch]
    uint32_t *w_ring = stage_all + kTcFoldWarps * 32 * kTcStagePitch;       // [depth][tap][KWC][kTcN] weight bit words
    uint32_t *p_ring = w_ring + a.depth * (KHW * KWC * kTcN);               // [depth][RA][KWC][256] patch bit words
    uint4 *bias_s = reinterpret_cast<uint4 *>(p_ring + a.depth * (RA * KWC * kTcExpandWarps * 32)); // [2][kTcUnit] pixel operand of 1s
    uint64_t *bars = reinterpret_cast<uint64_t *>(bias_s + 2 * kTcUnit);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + kTcBars);

    const int tid = threadIdx.x, lane = tid & 31;
    // the shuffle tells the compiler what it cannot see: the warp index is the same in every lane
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // Persistent CTA: it runs its tiles as ONE pipeline, so a tile's first loads / expansion and its last fold /
    // store overlap the neighbouring tiles' MMAs.  Its k-th tile is tile first_tile + k * tile_stride, of which it
    // computes time slots [slot_lo(k), slot_hi(k)): all of them, except in the first and last tile of a balanced run.
    // (The run is needed at tile switches only: it lives in shared memory, not in registers.)
    const TileRun &run = *reinterpret_cast<const TileRun *>(tmem_slot + 2);
    if (tid == 0)
        *reinterpret_cast<TileRun *>(tmem_slot + 2) = tile_run(a.total_tiles, a.slots, a.balanced, (int)blockIdx.x, (int)gridDim.x);
    auto slot_lo = [&](int k) { return k == 0 ? run.slot_first : 0; };
    auto slot_hi = [&](int k) { return k == run.tiles - 1 ? run.slot_last_end : a.slots; };
    auto tile_origin = [&](int k, long long &o0, int &nc) {
        const int L = run.first_tile + k * run.tile_stride;
        nc = L / a.tiles_x;                                  // 64-channel output chunk
        o0 = (long long)(L - nc * a.tiles_x) * kTcM;         // first candidate of the tile
    };

    // mbarriers (index = operand buffer b or unit u):
    //   full[b]   operands of a step are written                         (one arrival per expanding warp)
    //   empty[b]  the MMAs that read operand buffer b have completed     (one commit per step)
    //   done[u]   unit u's counts of a slot are complete                 (one commit per slot)
    //   tfree[u]  unit u's accumulators have been read                   (one arrival per folding warp)
    //   drain     every MMA has completed                                (one commit, at the issuing warp's exit)
    //   wfull[d]  the weight bit words of a step are in ring entry d     (bytes of the copies)
    //   wfree[d]  they have been expanded                                (one arrival per expanding warp)
    uint64_t *bar_full = bars, *bar_empty = bars + 2, *bar_tfree = bars + 4, *bar_done = bars + 6, *bar_drain = bars + 8;
    uint64_t *bar_wfull = bars + 9, *bar_wfree = bars + 9 + kTcMaxDepth;
    if (tid == 0) {
        auto init = [](uint64_t *bar, uint32_t count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
        };
        init(bar_drain, 1u);
        for (int b = 0; b < 2; b++) {
            init(&bar_full[b], kTcExpandWarps);
            init(&bar_empty[b], 1u);
            init(&bar_done[b], 1u);
            init(&bar_tfree[b], kTcFoldWarps / 2);
        }
        for (int d = 0; d < kTcMaxDepth; d++) {
            init(&bar_wfull[d], 1u);
            init(&bar_wfree[d], kTcExpandWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        // the whole tensor memory of the SM.  The allocation
        // blocks until all 512 columns are free, so this kernel assumes it is the only user of tensor memory on its
        // SM: its > 113 KB of dynamic shared memory keeps a second CTA of itself away, but a kernel of ANOTHER stream
        // that holds tensor memory (the FXP conv of this library, a vendor GEMM) would make the allocation wait for
        // that kernel's CTA to finish.  Callers that overlap streams must serialise this kernel with such kernels.
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                     "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t lane_quarter = (uint32_t)((warp & 3) * 32) << 16; // the TMEM lanes this warp can access
    if (warp < 4) {
        // block scales (biased exponents, the same in every byte, whatever row or block an MMA reads) and the weight
        // operand of the bias MMA
        auto fill = [&](uint32_t col, uint32_t v) {
            asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};"
                         ::"r"(tmem_base + lane_quarter + col), "r"(v) : "memory");
        };
        fill(kTcColSf, 0x7f7f7f7fu);
        fill(kTcColSf + 8, 0x7f7f7f7fu);
        fill(kTcColSfBias, 0x8a8a8a8au);
        fill(kTcColSfBias + 8, 0x8a8a8a8au);
        const uint32_t z = 0u, two = 4u; // e2m1 2.0 in the lowest nibble
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %2, %2, %2, %2, %2, %2};"
                     ::"r"(tmem_base + lane_quarter + kTcColBias), "r"(two), "r"(z) : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < 2 * kTcUnit; i += kTcThreads) bias_s[i] = make_uint4(0x22222222u, 0x22222222u, 0x22222222u, 0x22222222u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int total_steps = run.slots * a.CK; // pipeline steps of this CTA; slots are numbered through all of its tiles
    bool failed = false;
    // The warps run unsynchronised; every dependence is an mbarrier phase.  Phase parities: barrier index b is used
    // by steps b, b + 2, ... (done, tfree: by every slot); its k-th completion has parity k & 1.  A timed-out wait ends
    // the warp's loop; the warps that depend on it time out in turn, so everybody reaches the end of the kernel.
    auto wait_on = [&](uint64_t *bar, int k) {
        const bool ok = tc_wait(saddr(bar), (uint32_t)(k & 1));
        return __all_sync(0xffffffffu, ok) != 0;
    };
    auto warp_arrive = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
    };

    // one step further in a ring of a.depth entries; `round` counts the passes through it
    auto ring_next = [&](int &d, int &round) {
        if (++d == a.depth) { d = 0; round++; }
    };

    if (warp >= kTcIssueWarp) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsIssuer));
    if (warp == kTcIssueWarp) {
        // ---- MMA-issuing warp: operands ready -> accumulator free -> issue -> commit ----
        // The loop is kept to a few instructions per MMA: fully unrolled over taps, per-tap operand offsets in
        // registers, descriptors patched in their low word (the start-address field counts 16-byte units, i.e. operand
        // rows, from bit 0; no carry leaves the field because shared memory ends below 256 KB).
        // instruction descriptor: e2m1 operands (both K-major), ue8m0 block scales, N = 160, M = 128
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(kTcUnit >> 3) << 17) | (1u << 23) | ((uint32_t)(kTcN >> 4) << 24);
        uint32_t p_tap[kTcMaxTaps];
#pragma unroll
        for (int tap = 0; tap < kTcMaxTaps; tap++) p_tap[tap] = tap < KHW ? (uint32_t)a.tap_off[tap] : 0u;
        const uint64_t dp_proto = desc_interleaved(saddr(smem), (uint32_t)a.rows_a * 16);
        const uint32_t dp_hi = (uint32_t)(dp_proto >> 32);
        const uint64_t db_bias = desc_interleaved(saddr(bias_s), kTcUnit * 16);
        const uint32_t sf = tmem_base + kTcColSf;
        auto commit = [&](uint64_t *bar) { // arrives on the barrier when every MMA issued so far has completed
            asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                         "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(saddr(bar))
                         : "memory");
        };
        auto issue_unit = [&](int buf, int u, int ck) {
            const uint32_t dp_lo = (uint32_t)dp_proto + (uint32_t)buf * (a_bytes >> 4) + (uint32_t)(u * kTcUnit);
            const uint32_t w_lo = tmem_base + kTcColA + (uint32_t)(buf * kTcMaxWords * kTcWordCols);
            const uint32_t d_addr = tmem_base + (uint32_t)(u * kTcUnit);
            const int words = a.CW - ck * KWC; // words left in this chunk; an odd last one is paired with a zero word
            auto mma = [&](uint32_t wcol, uint32_t plo, uint32_t phi, uint32_t scales, uint32_t accumulate) {
                asm volatile(
                    "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t"
                    "mov.b64 db, {%2, %3};\n\t"
                    "setp.ne.b32 p, %5, 0;\n\t"
                    "elect.sync _|e, 0xffffffff;\n\t"
                    "@e tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], db, %4, [%6], [%6], p;\n\t}"
                    ::"r"(d_addr), "r"(wcol), "r"(plo), "r"(phi), "r"(idesc), "r"(accumulate), "r"(scales)
                    : "memory");
            };
            // a slot starts at 2^23 = (1 * 2^11) * (2 * 2^11): the counts then are the low bits of the accumulators
            if (ck == 0) mma(tmem_base + kTcColBias, (uint32_t)db_bias, (uint32_t)(db_bias >> 32), tmem_base + kTcColSfBias, 0u);
#pragma unroll
            for (int tap = 0; tap < (KHW_T ? KHW_T : kTcMaxTaps); tap++) {
                if (KHW_T || tap < a.KHW) {
#pragma unroll
                    for (int k = 0; k < KWC; k += 2) {
                        if (k > 0 && k >= words) break;
                        const uint32_t plo = dp_lo + p_tap[tap] + (uint32_t)k * (uint32_t)a.rows_a;
                        const uint32_t wcol = w_lo + (uint32_t)((tap * KWC + k) * kTcWordCols);
                        mma(wcol, plo, dp_hi, sf, 1u);
                    }
                }
            }
        };
        int s = 0, ck = 0; // slot (counted through all tiles) and chunk of the step
        for (int step = 0; step < total_steps; step++) {
            if (!wait_on(&bar_full[step & 1], step >> 1)) { failed = true; break; }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (ck == 0 && s > 0 && !wait_on(&bar_tfree[u], s - 1)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                issue_unit(step & 1, u, ck);
                if (ck == a.CK - 1) commit(&bar_done[u]);
            }
            if (failed) break;
            commit(&bar_empty[step & 1]);
            if (++ck == a.CK) { ck = 0; s++; }
        }
        // Whatever way the loop ended: arrive on the drain barrier once all MMAs this warp has issued are complete,
        // so that tensor memory is not released under an MMA still in flight after a timed-out wait.
        commit(bar_drain);
    } else if (warp == kTcLoadWarp) {
        // ---- loading warp: weight bit words -> ring, up to a.depth steps ahead ----
        const int my_tiles = run.tiles;
        int d = 0, round = 0, issued = 0;
        for (int k = 0; k < my_tiles && !failed; k++) {
            long long o0;
            int nc;
            tile_origin(k, o0, nc);
            for (int slot = slot_lo(k); slot < slot_hi(k) && !failed; slot++) {
                const uint32_t *src = Wb + ((size_t)nc * a.slots + slot) * kTcN * (size_t)(KHW * a.CW);
                for (int ck = 0; ck < a.CK; ck++, issued++) {
                    if (round > 0 && !wait_on(&bar_wfree[d], round - 1)) { failed = true; break; }
                    if (lane == 0) {
                        const int words = a.CW - ck * KWC < KWC ? a.CW - ck * KWC : KWC; // of the chunk
                        const uint32_t bytes = (uint32_t)words * kTcN * 4, bar = saddr(&bar_wfull[d]);
                        const uint32_t dst = saddr(w_ring + d * (KHW * KWC * kTcN));
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes * (uint32_t)KHW) : "memory");
                        auto copy = [&](uint32_t to, const uint32_t *from, uint32_t n) {
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                         ::"r"(to), "l"(from), "r"(n), "r"(bar) : "memory");
                        };
                        if (a.CW == KWC) copy(dst, src, bytes * (uint32_t)KHW); // the slot's words are one run
                        else
                            for (int tap = 0; tap < KHW; tap++)
                                copy(dst + (uint32_t)(tap * KWC * kTcN * 4), src + ((size_t)tap * a.CW + ck * KWC) * kTcN, bytes);
                    }
                    __syncwarp();
                    ring_next(d, round);
                }
            }
        }
        // no copy may still be on its way when the CTA exits (after a time-out; otherwise all have been consumed)
        for (int j = issued > a.depth ? issued - a.depth : 0; j < issued; j++)
            if (!wait_on(&bar_wfull[j % a.depth], j / a.depth)) failed = true;
    } else if (warp >= kTcIssueWarp) {
        // (idle)
    } else if (warp >= kTcFoldWarps) {
        // ---- expanding warps: bit words -> operands ----
        // Two warps per TMEM lane quarter: they share a weight row's words (even ones, odd ones) and the patch rows.
        //   weights: row = this thread's TMEM lane, words read from the loading warp's ring
        //   patch:   row g = et + 256 * r of the residue planes; every thread copies its own rows' words into its own
        //            places of the ring, a.depth - 1 steps ahead, with asynchronous 4-byte copies (zeros where there is
        //            no pixel or no channel).  The copies walk the steps in order, the step-dependent part of every
        //            address is a running pointer.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsExpand));
        constexpr int kTaps = KHW_T ? KHW_T : kTcMaxTaps, kRows = kTcExpandWarps * 32;
        const int et = tid - kTcFoldWarps * 32, w_row = et & (kTcN - 1), w_par = (warp >> 2) & 1;
        const int my_tiles = run.tiles;
        const uint32_t *a_plane = Ab;
        uint32_t a_off[RA]; // stored-grid position of the thread's patch rows, ~0u: outside the tensor
        int ld_ck = 0, ld_left = 0, ld_tile = -1, ld_d = 0;
        // point the loads at the first slot and chunk of tile k of this CTA
        auto load_tile = [&](int k) {
            long long o0;
            int nc;
            tile_origin(k, o0, nc);
            const int slot0 = slot_lo(k);
            ld_tile = k;
            ld_ck = 0;
            ld_left = (slot_hi(k) - slot0) * a.CK;
            a_plane = Ab + (size_t)slot0 * a.CW * a.NHWp;                   // bit plane of the first slot, word 0
#pragma unroll
            for (int r = 0; r < RA; r++) {
                const int g = et + kRows * r;
                a_off[r] = ~0u;
                if (g < a.rows_a) {
                    const int plane = g / a.Mh, q = g - plane * a.Mh;
                    // candidate indices fit 31 bits (checked on the host); rows before the first stored pixel wrap
                    // around to large values and are zero like the rows behind the last one
                    const uint32_t o = (uint32_t)o0 + (uint32_t)q - (uint32_t)a.shift;
                    if (o < (uint32_t)a.total_o) {
                        const uint32_t t = o / (uint32_t)a.Wo, j = o - t * (uint32_t)a.Wo;
                        const uint32_t n = t / (uint32_t)a.Ho, i = t - n * (uint32_t)a.Ho;
                        const int rh = plane / a.nrw, rw = plane - rh * a.nrw;
                        a_off[r] = (n * (uint32_t)a.Hrows + i * (uint32_t)a.nrh + (uint32_t)rh) * (uint32_t)a.Wrow +
                                   (uint32_t)(rw * a.Wq) + j; // < NHWp < 2^32
                    }
                }
            }
        };
        // start the copies of the next step (none behind the last one: the group is then empty)
        auto load_bits = [&]() {
            if (ld_left > 0) {
                const int words_left = a.CW - ld_ck * KWC; // words of this chunk that exist; the others are zero
                const uint32_t dst0 = saddr(p_ring + ld_d * (RA * KWC * kRows) + et);
#pragma unroll
                for (int r = 0; r < RA; r++)
#pragma unroll
                    for (int k = 0; k < KWC; k++) {
                        const bool ok = a_off[r] != ~0u && k < words_left;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst0 + (uint32_t)((r * KWC + k) * kRows * 4)),
                                     "l"(ok ? a_plane + (size_t)k * a.NHWp + a_off[r] : Ab), "r"(ok ? 4 : 0) : "memory");
                    }
                // advance: next chunk of the slot, or chunk 0 of the next slot
                if (++ld_ck == a.CK) {
                    ld_ck = 0;
                    a_plane += (size_t)(a.CW - KWC * (a.CK - 1)) * a.NHWp;
                } else {
                    a_plane += (size_t)KWC * a.NHWp;
                }
                if (--ld_left == 0 && ld_tile + 1 < my_tiles) load_tile(ld_tile + 1); // the next call fetches the next tile
                if (++ld_d == a.depth) ld_d = 0;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const uint32_t w_dst0 = tmem_base + kTcColA + lane_quarter + (uint32_t)(w_par * kTcWordCols);
        const uint32_t a_kcol = (uint32_t)a.rows_a * 16;
        auto expand_bits = [&](int buf, int d, int words) { // words: of this chunk; an odd last one gets a zero partner
            const uint32_t w_dst = w_dst0 + (uint32_t)(buf * kTcMaxWords * kTcWordCols);
            const uint32_t *w_src = w_ring + d * (KHW * KWC * kTcN) + w_par * kTcN + w_row;
            const uint32_t *p_src = p_ring + d * (RA * KWC * kRows) + et;
            uint8_t *a_s = smem + (uint32_t)buf * a_bytes + (uint32_t)et * 16;
#pragma unroll
            for (int tap = 0; tap < kTaps; tap++) {
                if (KHW_T || tap < KHW) {
#pragma unroll
                    for (int k = 0; k < KWC; k += 2) {
                        const uint4 v = spread_weights(k + w_par < words ? w_src[(tap * KWC + k) * kTcN] : 0u);
                        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(w_dst + (uint32_t)((tap * KWC + k) * kTcWordCols)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RA; r++) {
                if (et + kRows * r < a.rows_a) {
                    uint8_t *dst = a_s + r * (kRows * 16);
#pragma unroll
                    for (int k = 0; k < KWC; k++)
                        *reinterpret_cast<uint4 *>(dst + k * a_kcol) = spread_pixels(p_src[(r * KWC + k) * kRows]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        };
        load_tile(0);
        for (int i = 0; i < a.depth - 1; i++) load_bits();
        int ck = 0, d = 0, round = 0;
        for (int step = 0; step < total_steps; step++) {
            load_bits(); // a.depth - 1 steps ahead; its ring entry is the one this thread emptied in the step before
            if (a.depth == kTcMaxDepth) asm volatile("cp.async.wait_group %0;" ::"n"(kTcMaxDepth - 1) : "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (!wait_on(&bar_wfull[d], round)) { failed = true; break; }
            if (step >= 2) { // the MMAs that read this buffer two steps ago
                if (!wait_on(&bar_empty[step & 1], (step >> 1) - 1)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            expand_bits(step & 1, d, a.CW - ck * KWC);
            warp_arrive(&bar_full[step & 1]);
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(&bar_wfree[d])) : "memory");
            ring_next(d, round);
            if (++ck == a.CK) ck = 0;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ---- folding warps: counts -> min(count, n) -> running sums -> outputs ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcRegsFold));
        // Warps 0-7 fold unit 0 while the tensor core is on unit 1, warps 8-15 the other way round.  This thread owns one
        // weight row (lane 32*(warp%4)+lane = sign and output channel) and kTcCols candidates of its unit, two 16-bit
        // sums per register.
        uint32_t sum[kTcCols / 2];
#pragma unroll
        for (int j = 0; j < kTcCols / 2; j++) sum[j] = 0u;
        const int u = warp >> 3, col0 = ((warp >> 2) & 1) * kTcCols; // unit, first column of the warp in it
        const uint32_t taddr = tmem_base + lane_quarter + (uint32_t)(u * kTcUnit + col0);
        const uint32_t n2 = (uint32_t)a.n_or * 0x00010001u;
        // The accumulators are 2^23 + count, so the packed read delivers two integer counts per register.  All of them
        // are read at once and handed back before the arithmetic: the unit's next MMAs wait for one TMEM read.
        auto fold_slot = [&]() {
            uint32_t x0[16], x1[16], x2[8];
            REXSC_TMEM_LD32P(x0, taddr);
            REXSC_TMEM_LD32P(x1, taddr + 32u);
            REXSC_TMEM_LD16P(x2, taddr + 64u);
            REXSC_TMEM_WAIT16(x0);
            REXSC_TMEM_WAIT16(x1);
            REXSC_TMEM_WAIT8(x2);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            warp_arrive(&bar_tfree[u]);
#pragma unroll
            for (int j = 0; j < 16; j++) sum[j] += __vminu2(x0[j], n2);
#pragma unroll
            for (int j = 0; j < 16; j++) sum[16 + j] += __vminu2(x1[j], n2);
#pragma unroll
            for (int j = 0; j < 8; j++) sum[32 + j] += __vminu2(x2[j], n2);
        };
        static_assert(kTcCols == 80, "fold_slot reads 32 + 32 + 16 columns");
        // Running sums -> int16 outputs, after the last slot of tile k.  A warp holds 32 output channels of one sign x
        // kTcCols candidates; they pass through its staging rows, 32 at a time, so that stores run along channels
        // (channels_last) or along pixels (channel-planar).  A candidate (i, j) of the origin grid is an output pixel
        // iff i < OH and j < OW.
        uint32_t *stage = stage_all + warp * (32 * kTcStagePitch);
        const uint16_t *stage16 = reinterpret_cast<const uint16_t *>(stage);
        auto store_tile = [&](int k) {
            long long o0;
            int nc;
            tile_origin(k, o0, nc);
            const bool shared_tile = slot_hi(k) - slot_lo(k) < a.slots; // other CTAs hold the tile's other time slots
            const int row0 = (warp & 3) * 32;
            const int co0 = nc * kTcCout + (row0 & (kTcCout - 1));     // channel of the warp's first row
            int16_t *dst = row0 >= kTcCout ? out_neg : out_pos;
            const size_t ohw = (size_t)a.OH * a.OW;
#pragma unroll
            for (int h = 0; h < kTcCols; h += kTcStageCols) {
                constexpr int kS = kTcStageCols;
                const int cnt = kTcCols - h < kS ? kTcCols - h : kS;
                __syncwarp();
#pragma unroll
                for (int j = 0; j < kS / 2; j++) {
                    if (h / 2 + j >= kTcCols / 2) break;
                    stage[lane * kTcStagePitch + j] = sum[h / 2 + j];
                    sum[h / 2 + j] = 0u;
                }
                __syncwarp();
                // lane l decodes candidate h + l: element of channel 0, -1: no output pixel
                long long base = -1;
                const uint32_t o = (uint32_t)o0 + (uint32_t)(u * kTcUnit + col0 + h + lane);
                if (lane < cnt && o < (uint32_t)a.total_o) {
                    const uint32_t t = o / (uint32_t)a.Wo, n = t / (uint32_t)a.Ho;
                    const int ow = (int)(o - t * (uint32_t)a.Wo), oh = (int)(t - n * (uint32_t)a.Ho);
                    if (ow < a.OW && oh < a.OH) {
                        const size_t pix = (size_t)oh * a.OW + ow;
                        base = (long long)(a.out_nhwc ? ((size_t)n * ohw + pix) * a.Co : (size_t)n * a.Co * ohw + pix);
                    }
                }
                if (a.balanced != 2 && a.out_nhwc && a.out_vec && !shared_tile) {
                    // eight channels per lane, eight pixels at a time
                    const int c8 = (lane & 3) * 8;
#pragma unroll 2
                    for (int p = lane >> 2; p < cnt; p += 8) {
                        const long long b = __shfl_sync(0xffffffffu, base, p);
                        uint32_t v[4];
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            v[q] = (uint32_t)stage16[(c8 + 2 * q) * (2 * kTcStagePitch) + p] |
                                   ((uint32_t)stage16[(c8 + 2 * q + 1) * (2 * kTcStagePitch) + p] << 16);
                        if (b >= 0 && co0 + c8 < a.Co)
                            *reinterpret_cast<uint4 *>(dst + b + co0 + c8) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                } else if (a.balanced != 2 && a.out_nhwc && a.out_al4 && (a.Co & 1) == 0) {
                    // two channels per lane, two pixels per store
                    const int w = lane & 15;
#pragma unroll 4
                    for (int p = lane >> 4; p < cnt; p += 2) {
                        const long long b = __shfl_sync(0xffffffffu, base, p);
                        if (b >= 0 && co0 + 2 * w < a.Co) {
                            const uint32_t v = (uint32_t)stage16[(2 * w) * (2 * kTcStagePitch) + p] |
                                               ((uint32_t)stage16[(2 * w + 1) * (2 * kTcStagePitch) + p] << 16);
                            uint32_t *q = reinterpret_cast<uint32_t *>(dst + b + co0 + 2 * w);
                            // partial sums of this share of the slots: two int16 per 32-bit add, no carry can cross
                            // the halves because the complete sums fit 16 bits (the host cuts tiles for aligned rows only)
                            if (shared_tile) atomicAdd(q, v);
                            else *q = v;
                        }
                    }
                } else {
                    // One value per lane.  balanced == 2: EVERY tile of the launch adds its sums into outputs that the
                    // host cleared, one 16-bit value per 32-bit atomic add on the word that holds it (no carry leaves
                    // the value's half: the complete sums fit 16 bits; the word's other half gets + 0).  All accesses to
                    // these words are atomic adds, so neighbours stored by other CTAs cannot be lost.
                    auto put = [&](long long e, uint32_t v) {
                        if (a.balanced == 2) {
                            if (v != 0u) {
                                const uintptr_t addr = reinterpret_cast<uintptr_t>(dst + e);
                                atomicAdd(reinterpret_cast<unsigned int *>(addr & ~(uintptr_t)3), v << ((addr & 2u) * 8u));
                            }
                        } else {
                            dst[e] = (int16_t)v;
                        }
                    };
                    if (a.out_nhwc) {
#pragma unroll 4
                        for (int p = 0; p < cnt; p++) { // lane = channel
                            const long long b = __shfl_sync(0xffffffffu, base, p);
                            if (b >= 0 && co0 + lane < a.Co) put(b + co0 + lane, stage16[lane * (2 * kTcStagePitch) + p]);
                        }
                    } else { // lane = candidate; half a group of candidates leaves room for two channels
                        const int rows = 32 / cnt, p = lane % cnt;
                        const long long b = __shfl_sync(0xffffffffu, base, p);
#pragma unroll 4
                        for (int r = lane / cnt; r < 32; r += rows)
                            if (b >= 0 && co0 + r < a.Co)
                                put(b + (long long)((size_t)(co0 + r) * ohw), stage16[r * (2 * kTcStagePitch) + p]);
                    }
                }
            }
        };
        int s = 0; // slot, counted through all tiles
        for (int k = 0; k < run.tiles && !failed; k++) {
            const int n_slots = slot_hi(k) - slot_lo(k);
            for (int i = 0; i < n_slots && !failed; i++, s++) {
                if (!wait_on(&bar_done[u], s)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                fold_slot();
                if (i == n_slots - 1) store_tile(k);
            }
        }
    }
    if (failed && lane == 0) atomicExch(status, 4);
    // (a warp whose wait timed out leaves its share of the remaining tiles unwritten; the status word reports it)

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        // bounded like every other wait; in a run without time-outs the MMAs are long complete and this returns at once
        if (!wait_on(bar_drain, 0) && lane == 0) atomicExch(status, 4);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// Zeroes the output rows of every tile that two CTAs of a balanced launch share (see TcArgs::balanced).  Block b looks
// at the cut between runs b and b + 1; a cut inside a tile makes that tile shared.  `grid` is the conv launch's grid.
__global__ void __launch_bounds__(kTcM)
zero_shared_tiles_kernel(TcArgs a, int grid, int16_t *__restrict__ out_pos, int16_t *__restrict__ out_neg,
                         const int *__restrict__ status, int gate)
{
    if (gate != 0 && (gate > 0) == (status[1] != 0)) return;
    const long long units = (long long)a.total_tiles * a.slots;
    const long long cut = units * ((int)blockIdx.x + 1) / grid;
    if (cut % a.slots == 0) return;
    const int L = (int)(cut / a.slots), nc = L / a.tiles_x;
    const uint32_t o0 = (uint32_t)(L - nc * a.tiles_x) * kTcM;
    // One row (candidate) per thread decodes its output position; then the warp writes its 32 rows one after the other,
    // lane l the l-th of the row's 32 words of each sign (rows are 4-byte aligned and hold whole 64-channel chunks, or
    // the host would not have cut tiles).
    const int lane = threadIdx.x & 31;
    const uint32_t o = o0 + threadIdx.x; // blockDim.x == kTcM
    long long word0 = -1;                // first 32-bit word of the row, -1: the candidate is no output pixel
    if (o < (uint32_t)a.total_o) {
        const uint32_t t = o / (uint32_t)a.Wo, n = t / (uint32_t)a.Ho;
        const int ow = (int)(o - t * (uint32_t)a.Wo), oh = (int)(t - n * (uint32_t)a.Ho);
        if (ow < a.OW && oh < a.OH)
            word0 = (long long)(((((size_t)n * a.OH + oh) * a.OW + ow) * a.Co + (size_t)nc * kTcCout) / 2);
    }
    uint32_t *pos32 = reinterpret_cast<uint32_t *>(out_pos), *neg32 = reinterpret_cast<uint32_t *>(out_neg);
#pragma unroll 4
    for (int j = 0; j < 32; j++) {
        const long long w = __shfl_sync(0xffffffffu, word0, j);
        if (w >= 0) {
            pos32[w + lane] = 0u;
            neg32[w + lane] = 0u;
        }
    }
}

// Tensor-pipe issue-rate probe: back-to-back int8 MMAs (M128 x N x K32) on fixed shared-memory operands.
__global__ void __launch_bounds__(128, 2) mma_probe_kernel(int iters, int n_cols, uint32_t *sink)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((128u - (saddr(smem_raw) & 127u)) & 127u);
    uint8_t *a_s = smem;                 // [2][128][16]
    uint8_t *b_s = smem + 2 * 128 * 16;  // [2][n_cols][16]
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < (2 * 128 * 16 + 2 * n_cols * 16) / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_slot)),
                     "r"((uint32_t)n_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n_cols >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    bool ok = true;
    if (tid == 0) {
        const uint64_t da = desc_interleaved(saddr(a_s), 128 * 16), db = desc_interleaved(saddr(b_s), (uint32_t)n_cols * 16);
        uint32_t phase = 0;
        for (int it = 0; it < iters && ok; it++) {
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const uint32_t accumulate = (it > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                    ::"r"(tmem_base), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
                    : "memory");
            }
            // commit and wait every 64 iterations so that the queue stays full but bounded
            if ((it & 63) == 63 || it == iters - 1) {
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(&bar))
                             : "memory");
                ok = tc_wait(saddr(&bar), phase & 1u);
                phase++;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t v[8];
    REXSC_TMEM_LD16P(v, tmem_base + ((uint32_t)(warp * 32) << 16));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    sink[blockIdx.x * blockDim.x + tid] = v[0] + (ok ? 0u : 0x80000000u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)n_cols) : "memory");
}

// geometry of the tensor-core kernel for one plan; ok = false when the layer does not fit
struct TcGeom {
    bool ok;
    int planes, Ho, Wo, Mh, rows_a, KWc, CK, CW, ra, depth;
    size_t smem;
    int tap_off[kTcMaxTaps];
};

TcGeom tc_geometry(const ConvPlan &p)
{
    TcGeom g{};
    g.ok = false;
    if (p.KHW > kTcMaxTaps || p.KHW < 1) return g;
    g.planes = p.nrh * p.nrw;
    g.Ho = p.Hrows / p.nrh;
    g.Wo = p.Wq;
    int max_shift = 0;
    for (int kh = 0; kh < p.KH; kh++)
        for (int kw = 0; kw < p.KW; kw++) {
            const int shift = (kh / p.sh) * g.Wo + kw / p.sw;
            if (shift > max_shift) max_shift = shift;
        }
    g.Mh = (kTcM + max_shift + 7) / 8 * 8;
    g.rows_a = g.planes * g.Mh;
    static_assert((kTcM - kTcPlaneTile) % 8 == 0, "Mh is rounded to 8 rows");
    if (g.planes * (g.Mh - (kTcM - kTcPlaneTile)) > kTcMaxPlaneRows) return g;
    if (g.rows_a > kTcMaxARows * (kTcExpandWarps * 32)) return g;
    for (int t = 0; t < kTcMaxTaps; t++) g.tap_off[t] = 0;
    for (int kh = 0; kh < p.KH; kh++)
        for (int kw = 0; kw < p.KW; kw++) {
            const int plane = (kh % p.sh) * p.nrw + kw % p.sw; // residues below nrh / nrw by construction of the grid
            g.tap_off[kh * p.KW + kw] = plane * g.Mh + (kh / p.sh) * g.Wo + kw / p.sw;
        }
    g.CW = (p.C + 31) / 32;
    // Words per pipeline step: two (one MMA per tap and unit), and for 1x1 filters, whose steps are short, as many as
    // the layer has up to eight.
    g.KWc = p.KHW == 1 ? (g.CW <= 2 ? 2 : g.CW <= 4 ? 4 : 8) : 2;
    if (p.KHW * g.KWc > kTcMaxWords) return g;
    g.CK = (g.CW + g.KWc - 1) / g.KWc;
    g.ra = (g.rows_a + kTcExpandWarps * 32 - 1) / (kTcExpandWarps * 32);
    g.ra = p.KHW == 1 || g.ra <= 2 ? 2 : g.ra <= 6 ? 6 : kTcMaxARows; // the instantiated row counts
    auto need = [&](int depth) {
        return 2 * (size_t)g.KWc * g.rows_a * 16 + (size_t)kTcFoldWarps * 32 * kTcStagePitch * 4 +
               (size_t)depth * g.KWc * 4 * (p.KHW * kTcN + g.ra * kTcExpandWarps * 32) + 2 * kTcUnit * 16 + kTcBars * 8 + 8 +
               sizeof(TileRun) + 128;
    };
    g.depth = need(kTcMaxDepth) <= 227 * 1024 ? kTcMaxDepth : 2;
    if (need(g.depth) > 227 * 1024) return g;
    // the kernel owns the SM's whole tensor memory: ask for enough shared memory that no second CTA is co-scheduled
    g.smem = need(g.depth) > 120 * 1024 ? need(g.depth) : 120 * 1024;
    g.ok = true;
    return g;
}

} // namespace

int launch_mma_probe(int blocks, int iters, int n_cols, uint32_t *d_sink, cudaStream_t st)
{
    if (blocks < 1 || iters < 1 || (n_cols != 128 && n_cols != 256) || !d_sink) return REXSC_E_BAD_ARG;
    const size_t smem = 2 * 128 * 16 + 2 * (size_t)n_cols * 16 + 128;
    mma_probe_kernel<<<blocks, 128, smem, st>>>(iters, n_cols, d_sink);
    REXSC_LAUNCH_CHECK("mma_probe_kernel");
    return REXSC_OK;
}

bool conv_tc_supported(const ConvPlan &p)
{
    if (p.n_or < 1) return false;
    if (p.Hrows % p.nrh != 0) return false;
    const TcGeom g = tc_geometry(p);
    if (!g.ok) return false;
    const long long cap = p.n_or < p.Kdot ? p.n_or : p.Kdot;                   // largest per-slot contribution
    if ((long long)p.words * 32 * cap > 65535) return false;                  // 16-bit running sums
    // The packed read of 2^23 + count has room for counts up to 65535.  Longer dot products than 8191 have not been run on
    // this path and stay where they are, on the ALU kernels.
    if (p.Kdot > 8191) return false;
    const long long total_o = (long long)p.N * g.Ho * g.Wo;
    if (total_o + kTcM > 0x7fffffffLL) return false;                          // 31-bit candidate indices
    if ((total_o + kTcM - 1) / kTcM * ((p.Co + kTcCout - 1) / kTcCout) > 0x7fffffffLL) return false; // tile index: int
    if (p.NHWp > 0xfffffffeLL) return false;                                  // 32-bit position offsets
    return true;
}

size_t conv_tc_workspace_bytes(const ConvPlan &p)
{
    const int CW = (p.C + 31) / 32, NC = (p.Co + kTcCout - 1) / kTcCout;
    const size_t ab = (size_t)p.words * 32 * CW * p.NHWp * 4;
    const size_t wb = (size_t)NC * p.words * 32 * kTcN * p.KHW * CW * 4;
    return align_up(ab, 256) + align_up(wb, 256);
}

// byte offset of the weight bit planes Wb inside the tensor-core region of the workspace (Ab comes first)
size_t conv_tc_weight_offset(const ConvPlan &p)
{
    const int CW = (p.C + 31) / 32;
    return align_up((size_t)p.words * 32 * CW * p.NHWp * 4, 256);
}

static int device_sms(int *sms)
{
    int dev = 0;
    REXSC_CUDA_CHECK(cudaGetDevice(&dev));
    REXSC_CUDA_CHECK(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    return REXSC_OK;
}

// One persistent CTA per SM (the kernel owns the SM's tensor memory).  Whole tiles dealt round-robin leave SMs idle in
// the last wave (900 tiles on 148 SMs: 7 waves for the work of 6.1); cutting the (tile, slot) sequence into equal runs
// does not.  balanced: see TcArgs.
struct TcSplit { int balanced; unsigned grid; };

static TcSplit tc_split(const ConvPlan &p, const rexsc_sc_conv_desc &d, const int16_t *d_pos, const int16_t *d_neg, int gate,
                        int sms, long long total_tiles)
{
    TcSplit r{0, (unsigned)(total_tiles < sms ? total_tiles : sms)};
    static const bool allow_balanced = !(getenv("REXSC_TC_BALANCED") && getenv("REXSC_TC_BALANCED")[0] == '0');
    // The cut tiles are summed with packed 32-bit atomic adds, which need 4-byte aligned rows of whole 64-channel chunks;
    // the fallback launch of a gated pair keeps whole tiles (it is the rare one and a second clearing kernel would cost
    // every call).
    const bool aligned4 = ((reinterpret_cast<uintptr_t>(d_pos) | reinterpret_cast<uintptr_t>(d_neg)) & 3u) == 0;
    const bool rows_ok = d.out_channels_last && (p.Co % kTcCout) == 0 && aligned4;
    // (measured: tiles with little tensor work per slot -- 1x1 filters on up to 256 channels -- gain nothing: their
    // time goes to the per-slot hand-offs, and the atomic stores of the cut tiles cost more than the idle SMs did)
    const bool heavy_slots = p.KHW * ((p.C + 31) / 32) >= 16 || total_tiles < sms;
    if (!allow_balanced || !heavy_slots || !aligned4 || gate < 0 || total_tiles % sms == 0) return r;
    // Outputs without such rows (NCHW, a ragged last chunk): clear them whole and let every tile add single 16-bit
    // values -- affordable while the outputs are small, which is where whole tiles waste most (deep layers with few
    // tiles per SM).  The element count must be even so that the last value's 32-bit word ends inside the tensor.
    const size_t out_elems = (size_t)p.M * p.Co;
    if (!rows_ok && ((out_elems & 1) != 0 || out_elems * sizeof(int16_t) > ((size_t)16 << 20))) return r;
    // short layers: as many CTAs as leaves each about four slots to amortise its prologue
    long long ctas = total_tiles * p.words * 32 / 4;
    if (ctas < 1) ctas = 1;
    if (ctas > sms) ctas = sms;
    // worth a clearing launch when the last wave of whole tiles would waste more than 1 % (single values: 5 %) of the SM time
    const long long waves = (total_tiles + sms - 1) / sms;
    if ((double)total_tiles / sms < (rows_ok ? 0.99 : 0.95) * (double)waves || ctas > (long long)r.grid) {
        r.balanced = rows_ok ? 1 : 2;
        r.grid = (unsigned)ctas;
    }
    return r;
}

long long conv_tc_clear_words(const ConvPlan &p, const rexsc_sc_conv_desc &d, const int16_t *d_pos, const int16_t *d_neg)
{
    const size_t bytes = (size_t)p.M * p.Co * sizeof(int16_t);
    // 4 MB per sign are about 1 us of the expand launch; clearing the shared tiles alone is a launch of 4 us
    if (bytes > ((size_t)4 << 20) || (bytes & 15) != 0) return 0;
    if ((reinterpret_cast<uintptr_t>(d_pos) | reinterpret_cast<uintptr_t>(d_neg)) & 15u) return 0;
    int sms = 0;
    if (!conv_tc_supported(p) || device_sms(&sms) != REXSC_OK) return 0;
    const TcGeom g = tc_geometry(p);
    const long long tiles_x = ((long long)p.N * g.Ho * g.Wo + kTcM - 1) / kTcM;
    const TcSplit r = tc_split(p, d, d_pos, d_neg, 0, sms, tiles_x * ((p.Co + kTcCout - 1) / kTcCout));
    return r.balanced ? (long long)(bytes / 16) : 0;
}

int launch_conv_tc(const ConvPlan &p, const rexsc_sc_conv_desc &d, void *d_tc_ws, size_t weight_offset, int16_t *d_pos,
                   int16_t *d_neg, int *d_status, int gate, bool outputs_cleared, cudaStream_t st)
{
    if (!conv_tc_supported(p)) return REXSC_E_UNSUPPORTED;
    const TcGeom g = tc_geometry(p);
    const int CW = g.CW, NC = (p.Co + kTcCout - 1) / kTcCout;
    const int slots = p.words * 32;
    const uint32_t *Ab = static_cast<const uint32_t *>(d_tc_ws);
    const uint32_t *Wb = reinterpret_cast<const uint32_t *>(static_cast<const uint8_t *>(d_tc_ws) + weight_offset);
    TcArgs a;
    a.OH = p.OH; a.OW = p.OW; a.KHW = p.KHW; a.Co = p.Co;
    a.CW = CW; a.CK = g.CK; a.depth = g.depth;
    a.nrh = p.nrh; a.nrw = p.nrw; a.Wq = p.Wq; a.Hrows = p.Hrows; a.Wrow = p.Wrow;
    a.Ho = g.Ho; a.Wo = g.Wo; a.Mh = g.Mh; a.rows_a = g.rows_a;
    a.shift = p.origin ? g.Wo + 1 : 0;
    a.slots = slots;
    a.total_o = (long long)p.N * g.Ho * g.Wo;
    a.tiles_x = (int)((a.total_o + kTcM - 1) / kTcM);
    int sms = 0;
    if (int rc = device_sms(&sms)) return rc;
    a.total_tiles = a.tiles_x * NC;
    const bool aligned4 = ((reinterpret_cast<uintptr_t>(d_pos) | reinterpret_cast<uintptr_t>(d_neg)) & 3u) == 0;
    const TcSplit split = tc_split(p, d, d_pos, d_neg, gate, sms, a.total_tiles);
    const unsigned grid = split.grid;
    a.balanced = split.balanced;
    if (a.balanced == 2 && !outputs_cleared) {
        const size_t out_bytes = (size_t)p.M * p.Co * sizeof(int16_t);
        REXSC_CUDA_CHECK(cudaMemsetAsync(d_pos, 0, out_bytes, st));
        REXSC_CUDA_CHECK(cudaMemsetAsync(d_neg, 0, out_bytes, st));
    }
    if (a.balanced == 1 && grid > 1 && !outputs_cleared) {
        zero_shared_tiles_kernel<<<grid - 1, kTcM, 0, st>>>(a, (int)grid, d_pos, d_neg, d_status, gate);
        REXSC_LAUNCH_CHECK("zero_shared_tiles_kernel");
    }
    a.NHWp = p.NHWp; a.out_nhwc = d.out_channels_last;
    if ((reinterpret_cast<uintptr_t>(d_pos) | reinterpret_cast<uintptr_t>(d_neg)) & 1u) return REXSC_E_BAD_ARG;
    a.out_al4 = aligned4 ? 1 : 0;
    a.out_vec = ((reinterpret_cast<uintptr_t>(d_pos) | reinterpret_cast<uintptr_t>(d_neg)) & 15u) == 0 && (p.Co & 7) == 0 ? 1 : 0;
    {
        const long long cap = p.n_or < p.Kdot ? p.n_or : p.Kdot;
        a.n_or = (int)cap; // a count never exceeds the dot length, so clamping there changes nothing
    }
    for (int t = 0; t < kTcMaxTaps; t++) a.tap_off[t] = g.tap_off[t];
    auto kernel = p.KHW == 9 ? (g.ra == 2 ? sc_conv_tc_kernel<9, 2, 2> : g.ra == 6 ? sc_conv_tc_kernel<9, 2, 6> : sc_conv_tc_kernel<9, 2, kTcMaxARows>)
                : p.KHW != 1 ? (g.ra == 2 ? sc_conv_tc_kernel<0, 2, 2> : g.ra == 6 ? sc_conv_tc_kernel<0, 2, 6> : sc_conv_tc_kernel<0, 2, kTcMaxARows>)
                : g.KWc == 2 ? sc_conv_tc_kernel<1, 2, 2>
                : g.KWc == 4 ? sc_conv_tc_kernel<1, 4, 2> : sc_conv_tc_kernel<1, 8, 2>; // (one plane of kTcM rows)
    REXSC_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
    kernel<<<grid, kTcThreads, g.smem, st>>>(a, Ab, Wb, d_pos, d_neg, d_status, gate);
    REXSC_LAUNCH_CHECK("sc_conv_tc_kernel");
    return REXSC_OK;
}

} // namespace rexsc
