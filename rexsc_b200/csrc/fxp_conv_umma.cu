// FXP saturating conv, closed form, on the 5th-generation tensor cores (tcgen05, int8 -> int32 in TMEM).
//
// Valid exactly where fxp_conv.cu's closed form is (plain add, no shift, operands <= 127): per sign the
// reference's sequential saturating adder equals  min( sum a*w + sum (a&1)(w&1), 2^pmax ), every addend is
// non-negative, so splitting K into MMA steps cannot change where the sum saturates -- the cap is applied once to
// the finished int32 accumulator (the host checks that K*127*127 + K cannot overflow it).
//
// Implicit GEMM:  D[m][n'] = sum_k' A[m][k'] * B[n'][k'],  k' runs over the products twice (values, then parity
// bits), n' over the output channels of the CTA's chunk twice (positive weights, then negative weights).  CTA = 128
// output pixels (TMEM lanes) x up to 256 columns.  The products are ordered (tap, channel) with the channels padded
// to a multiple of 16 -- the order does not matter to the closed form -- and the int8 activations are kept pixel-major
// (NHWC, same channel padding), so 16 consecutive k' of an output pixel are 16 consecutive bytes in memory.
//   * k' is taken in slabs of 128 products; a pipeline step is a slab's values and, from the same registers, its
//     parity bits, so every activation is fetched once and a slab costs one hand-over to the tensor core;
//   * producers (all 128 threads): fetch the int8 activation slab (128 rows x 128 bytes of k') as eight 16-byte
//     loads per row through a chunk -> tensor-offset table, one step ahead (the table's entries two), and the prepacked
//     weight slabs with asynchronous copies (into the other of two buffers where a CTA has its SM to itself), both in the
//     128-byte swizzled K-major layout the MMA's shared-memory descriptors name;
//   * one thread issues tcgen05.mma.kind::i8 (M=128, N=N', K=32) eight times per step and commits to an mbarrier;
//   * epilogue: tcgen05.ld 32 lanes x 32 columns per warp, min(., cap), pos - neg, coalesced NCHW int32 stores.
// What bounds it: the latency of a step's gather, hand-over and MMAs, hidden by the other CTAs of the SM where there are
// enough.  TinyConv's four layers at batch 256, whole calls: 246 us with values and parity bits as separate slabs (every
// activation fetched twice, table entry and activation one after the other, weights through registers) and three
// launches, 155 us as it is.
// Every mbarrier wait is bounded; on a time-out the CTA records it, frees its TMEM and returns.
#include "common.cuh"
#include <type_traits>

namespace rexsc {

namespace {

constexpr int kUmmaM = 128;          // output pixels per CTA = TMEM lanes
constexpr int kSlabBytes = 128;      // k' bytes per pipeline step (one 128-byte swizzle row)
constexpr int kUmmaK = 32;           // int8 elements per MMA instruction
constexpr uint32_t kUmmaWaitLimit = 1u << 22;

struct UmmaArgs {
    int N, C, Hp, Wp, Co, OH, OW, sh, sw;
    int H, W, ph, pw; // unpadded activation and the op's zero padding (operand preparation)
    float scale;      // 2^precision_in
    int Cp;          // channels padded to 16 (pixel pitch of the int8 activations, channel pitch of k')
    int K2;          // products: taps x Cp
    int Kp;          // k' extent: per slab of products kSlabBytes of values, then kSlabBytes of parity bits
    int CB, CBp;     // output channels per CTA chunk, padded to 8
    int CBq;         // first MMA column of the negative-weight block (CBp rounded up to 32: aligned TMEM reads)
    int NP;          // MMA N: positive block [0, CBp), negative block [CBq, CBq + CBp), padded to 16
    int tmem_cols;   // power of two >= NP, >= 32
    int w_bufs;      // buffers of the weight slabs: 2 (those of the next step are copied during a step's MMAs) or 1
    int cap;
    long long M;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);       // start address, 16-byte units
    d |= (uint64_t)1 << 16;                       // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                       // descriptor version (Blackwell)
    d |= (uint64_t)2 << 61;                       // layout type: 128-byte swizzle
    return d;
}

// byte offset of 16-byte chunk `c` (0..7) of row `r` inside a [rows][128 B] tile with 128-byte swizzle
__device__ __forceinline__ uint32_t sw128_offset(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// Unswizzled ("interleaved") K-major alternative: the tile is stored as 16-byte K-columns, [chunk][row][16 B], so
// every row of a K-column sits 16 bytes after the previous one (8-row core matrices back to back, stride byte
// offset 128) and the next K-column starts `rows * 16` bytes later (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_k_interleaved(uint32_t saddr, uint32_t rows)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);
    d |= (uint64_t)(((rows * 16) >> 4) & 0x3fff) << 16; // leading byte offset: next 16-byte K-column
    d |= (uint64_t)(128 >> 4) << 32;                    // stride byte offset: next 8-row core matrix
    d |= (uint64_t)1 << 46;
    return d;                                           // layout type 0: no swizzle
}
__device__ __forceinline__ uint32_t interleaved_offset(int r, int c, int rows) { return (uint32_t)((c * rows + r) * 16); }

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t i = 0; i < kUmmaWaitLimit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

template <bool SWIZZLED>
__global__ void __launch_bounds__(128, 4)
fxp_conv_umma_kernel(UmmaArgs a, const int8_t *__restrict__ act, const int8_t *__restrict__ wpk,
                     const int32_t *__restrict__ koff, int32_t *__restrict__ out, int *__restrict__ status)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    // the swizzled operand tiles must start on a 1024-byte boundary of the shared window
    uint8_t *smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    const uint32_t a_tile = kUmmaM * kSlabBytes, b_tile = (uint32_t)((a.NP + 7) / 8 * 8) * kSlabBytes; // 1024-byte multiples
    uint8_t *a_s = smem;                                   // values, parity bits: 128 rows x 128 B each
    uint8_t *b_s = smem + 2 * a_tile;                      // [buffer][values, parity bits]: NP rows x 128 B each
    const int n_steps = a.Kp / (2 * kSlabBytes);
    uint64_t *bar = reinterpret_cast<uint64_t *>(b_s + 2 * a.w_bufs * b_tile);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const long long m = (long long)blockIdx.x * kUmmaM + tid;
    const int chunk = blockIdx.y;
    const bool row_live = m < a.M;
    long long abase = 0;
    int ow = 0, oh = 0, n = 0;
    if (row_live) {
        ow = (int)(m % a.OW);
        long long t = m / a.OW;
        oh = (int)(t % a.OH);
        n = (int)(t / a.OH);
        abase = (((long long)n * a.Hp + (long long)oh * a.sh) * a.Wp + (long long)ow * a.sw) * a.Cp;
    }

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    // instruction descriptor: int32 accumulate, signed int8 A and B, both K-major, N = NP, M = 128
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.NP >> 3) << 17) | ((uint32_t)(kUmmaM >> 4) << 24);
    const int8_t *wchunk = wpk + (size_t)chunk * a.NP * a.Kp;
    bool failed = false;

    // Row = this thread's output pixel, 8 chunks of 16 products each = 16 channels of one tap.  The chunks of step s + 1
    // are in flight while the tensor core works through step s, and so are its weight slabs; the table entries they are
    // fetched through are read another step earlier.
    // Of a last slab only the 32-product blocks that hold products are copied and multiplied (1, 2 or 4 of the 4).
    uint4 av[8];
    int off[8];
    auto log_blocks = [&](int step) {
        const int left = a.K2 - step * kSlabBytes;
        return left <= kUmmaK ? 0 : left <= 2 * kUmmaK ? 1 : 2;
    };
    auto load_off = [&](int step) {
#pragma unroll
        for (int c = 0; c < 8; c++) off[c] = step < n_steps ? __ldg(koff + step * 8 + c) : -1; // < 0: padding
    };
    auto load_act = [&]() {
#pragma unroll
        for (int c = 0; c < 8; c++) {
            av[c] = make_uint4(0u, 0u, 0u, 0u);
            if (row_live && off[c] >= 0) av[c] = __ldg(reinterpret_cast<const uint4 *>(act + abase + off[c]));
        }
    };
    auto load_weights = [&](int step) { // NP rows x 2 blocks of 16-byte chunks (values, then parity bits) -> buffer step & 1
        const uint32_t dst0 = smem_addr(b_s) + (uint32_t)(step & (a.w_bufs - 1)) * 2 * b_tile;
        const int lc = log_blocks(step) + 1; // log2 of the chunks of a row and half
        for (int e = tid; e < a.NP << (lc + 1); e += 128) {
            const int r = e >> (lc + 1), c = e & ((1 << lc) - 1), half = (e >> lc) & 1;
            const uint32_t dst = dst0 + (uint32_t)half * b_tile + (SWIZZLED ? sw128_offset(r, c) : interleaved_offset(r, c, a.NP));
            const int8_t *src = wchunk + (size_t)r * a.Kp + (size_t)step * 2 * kSlabBytes + half * kSlabBytes + c * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_weights(0);
    load_off(0);
    load_act();
    load_off(1);
    for (int step = 0; step < n_steps; step++) {
        const int blocks = 1 << log_blocks(step);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (c >= 2 * blocks) break;
            uint8_t *dst = a_s + (SWIZZLED ? sw128_offset(tid, c) : interleaved_offset(tid, c, kUmmaM));
            *reinterpret_cast<uint4 *>(dst) = av[c];
            *reinterpret_cast<uint4 *>(dst + a_tile) =
                make_uint4(av[c].x & 0x01010101u, av[c].y & 0x01010101u, av[c].z & 0x01010101u, av[c].w & 0x01010101u);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        // generic-proxy writes must be visible to the tensor core's async-proxy reads
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int half = 0; half < 2; half++) { // values, parity bits
                const uint32_t aa = smem_addr(a_s) + (uint32_t)half * a_tile;
                const uint32_t bb = smem_addr(b_s) + (uint32_t)((step & (a.w_bufs - 1)) * 2 + half) * b_tile;
                const uint64_t da = SWIZZLED ? umma_desc_k_sw128(aa) : umma_desc_k_interleaved(aa, kUmmaM);
                const uint64_t db = SWIZZLED ? umma_desc_k_sw128(bb) : umma_desc_k_interleaved(bb, a.NP);
#pragma unroll
                for (int kk = 0; kk < kSlabBytes / kUmmaK; kk++) {
                    if (kk >= blocks) break;
                    const uint32_t accumulate = (step > 0 || half > 0 || kk > 0) ? 1u : 0u;
                    // advancing K by 32 bytes: +2 address units (16 B) inside a swizzle row, or two K-columns further
                    // in the interleaved layout
                    const uint64_t dak = da + (uint64_t)(SWIZZLED ? kk * (kUmmaK >> 4) : kk * 2 * (kUmmaM * 16 >> 4));
                    const uint64_t dbk = db + (uint64_t)(SWIZZLED ? kk * (kUmmaK >> 4) : kk * 2 * (a.NP * 16 >> 4));
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                        ::"r"(tmem_base), "l"(dak), "l"(dbk), "r"(idesc), "r"(accumulate), "r"(0u)
                        : "memory");
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(bar))
                         : "memory");
        }
        if (step + 1 < n_steps) {
            if (a.w_bufs == 2) load_weights(step + 1); // (the MMAs of step - 1, which read that buffer, have completed)
            load_act();
            load_off(step + 2);
        }
        // the activation tiles are rewritten next step: wait until the MMAs that read them have completed
        if (!mbar_wait(smem_addr(bar), (uint32_t)(step & 1))) failed = true;
        failed = __syncthreads_or(failed ? 1 : 0) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (failed) break;
        if (a.w_bufs == 1 && step + 1 < n_steps) load_weights(step + 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    if (!failed) {
        // ---- epilogue: this warp reads its 32 TMEM lanes, 32 columns at a time ---------------------------------
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        const size_t ohw = (size_t)a.OH * a.OW;
        for (int c0 = 0; c0 < a.CBp; c0 += 32) {
            uint32_t vp[32], vn[32];
            const uint32_t tp = tmem_base + lane_base + (uint32_t)c0;
            const uint32_t tn = tmem_base + lane_base + (uint32_t)(a.CBq + c0);
            // both reads start on a multiple of 32 columns and stay inside the allocation (tmem_cols >= 2 * CBq);
            // columns at or past CB carry zero weights and are masked below
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(vp[0]), "=r"(vp[1]), "=r"(vp[2]), "=r"(vp[3]), "=r"(vp[4]), "=r"(vp[5]), "=r"(vp[6]), "=r"(vp[7]),
                  "=r"(vp[8]), "=r"(vp[9]), "=r"(vp[10]), "=r"(vp[11]), "=r"(vp[12]), "=r"(vp[13]), "=r"(vp[14]),
                  "=r"(vp[15]), "=r"(vp[16]), "=r"(vp[17]), "=r"(vp[18]), "=r"(vp[19]), "=r"(vp[20]), "=r"(vp[21]),
                  "=r"(vp[22]), "=r"(vp[23]), "=r"(vp[24]), "=r"(vp[25]), "=r"(vp[26]), "=r"(vp[27]), "=r"(vp[28]),
                  "=r"(vp[29]), "=r"(vp[30]), "=r"(vp[31])
                : "r"(tp) : "memory");
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(vn[0]), "=r"(vn[1]), "=r"(vn[2]), "=r"(vn[3]), "=r"(vn[4]), "=r"(vn[5]), "=r"(vn[6]), "=r"(vn[7]),
                  "=r"(vn[8]), "=r"(vn[9]), "=r"(vn[10]), "=r"(vn[11]), "=r"(vn[12]), "=r"(vn[13]), "=r"(vn[14]),
                  "=r"(vn[15]), "=r"(vn[16]), "=r"(vn[17]), "=r"(vn[18]), "=r"(vn[19]), "=r"(vn[20]), "=r"(vn[21]),
                  "=r"(vn[22]), "=r"(vn[23]), "=r"(vn[24]), "=r"(vn[25]), "=r"(vn[26]), "=r"(vn[27]), "=r"(vn[28]),
                  "=r"(vn[29]), "=r"(vn[30]), "=r"(vn[31])
                : "r"(tn) : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row_live) {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int cl = c0 + j;
                    const int co = chunk * a.CB + cl;
                    if (cl < a.CB && co < a.Co) {
                        const int p = min((int)vp[j], a.cap), q = min((int)vn[j], a.cap);
                        out[((size_t)n * a.Co + co) * ohw + (size_t)oh * a.OW + ow] = p - q;
                    }
                }
            }
        }
    } else if (tid == 0) {
        atomicExch(status, 3);
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)a.tmem_cols)
                     : "memory");
    }
}

// ---- operand preparation ------------------------------------------------------------------------------------
// One launch quantises on the fly (round-half-even of value * 2^p, fixed_cuda.cpp:28-30: activations clamped to
// [0, 2^p - 1], weights split into a positive and a negative magnitude): the first act_blocks blocks write the
// activations, the others the packed weights and the offset table.
// k' = slab by slab of 128 products tap * Cp + c: their values, then their parity bits; weights are [co][c][tap]
template <typename T>
__device__ __forceinline__ void pack_weights(const UmmaArgs &a, int KH, int KW, int n_chunks, const T *__restrict__ w,
                                             int8_t *__restrict__ wpk, int32_t *__restrict__ koff, int block, int blocks)
{
    const int KHW = KH * KW, K2 = KHW * a.Cp;
    // weights: wpk[chunk][row n' in 0..NP)[k' in 0..Kp), row = sign * CBq + local channel
    const long long total = (long long)n_chunks * a.NP * a.Kp;
    for (long long i = (long long)block * blockDim.x + threadIdx.x; i < total; i += (long long)blocks * blockDim.x) {
        const int kp = (int)(i % a.Kp);
        const long long r = i / a.Kp;
        const int row = (int)(r % a.NP);
        const int chunk = (int)(r / a.NP);
        const int sign = row >= a.CBq ? 1 : 0, cl = row - sign * a.CBq;
        const int co = chunk * a.CB + cl;
        const int slab = kp / (2 * kSlabBytes), in = kp - slab * 2 * kSlabBytes;
        const bool parity = in >= kSlabBytes;
        const int k = slab * kSlabBytes + (parity ? in - kSlabBytes : in);
        int v = 0;
        if (cl < a.CB && co < a.Co && k < K2) {
            const int tap = k / a.Cp, c = k - tap * a.Cp;
            if (c < a.C) {
                const float x = load_as_float<T>(w, ((long long)co * a.C + c) * KHW + tap) * a.scale;
                v = sign ? (int)rintf(-fminf(fmaxf(x, 1.f - a.scale), 0.f)) : (int)rintf(fminf(fmaxf(x, 0.f), a.scale - 1.f));
                if (parity) v &= 1;
            }
        }
        wpk[i] = (int8_t)v;
    }
    // 16-byte chunk of products -> byte offset of its 16 channels inside the int8 activations, relative to tap (0,0) of
    // the output pixel
    for (int j = block * blockDim.x + threadIdx.x; j < a.Kp / 32; j += blocks * blockDim.x) {
        const int k = j * 16;
        int off = -1;
        if (k < K2) {
            const int tap = k / a.Cp, cg = k - tap * a.Cp, kh = tap / KW, kw = tap - kh * KW;
            off = (kh * a.Wp + kw) * a.Cp + cg;
        }
        koff[j] = off;
    }
}

// dense NCHW activations -> zero-padded int8 NHWC with the channels padded to Cp; one thread per padded pixel and 16
// channels
template <typename TA, typename TW>
__global__ void __launch_bounds__(256) fxp_umma_prep_kernel(UmmaArgs a, int KH, int KW, int n_chunks, int act_blocks,
                                                            const TA *__restrict__ x, const TW *__restrict__ w,
                                                            int8_t *__restrict__ q8, int8_t *__restrict__ wpk,
                                                            int32_t *__restrict__ koff)
{
    if ((int)blockIdx.x >= act_blocks) {
        pack_weights<TW>(a, KH, KW, n_chunks, w, wpk, koff, (int)blockIdx.x - act_blocks, (int)gridDim.x - act_blocks);
        return;
    }
    const int groups = a.Cp / 16;
    const long long plane = (long long)a.Hp * a.Wp, total = (long long)a.N * plane * groups;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)act_blocks * blockDim.x) {
        // consecutive threads take consecutive pixels of one channel group: the strided reads coalesce
        const long long pix = i % plane;
        const long long t = i / plane;
        const int g = (int)(t % groups), n = (int)(t / groups);
        const int h = (int)(pix / a.Wp), wq = (int)(pix - (long long)h * a.Wp);
        const int hi = h - a.ph, wi = wq - a.pw;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (hi >= 0 && hi < a.H && wi >= 0 && wi < a.W) {
#pragma unroll
            for (int b = 0; b < 16; b++) {
                const int c = g * 16 + b;
                if (c < a.C) {
                    const float v = load_as_float<TA>(x, (((long long)n * a.C + c) * a.H + hi) * a.W + wi) * a.scale;
                    const int q = (int)rintf(fminf(fmaxf(v, 0.f), a.scale - 1.f));
                    w[b >> 2] |= (uint32_t)(q & 0xff) << (8 * (b & 3));
                }
            }
        }
        *reinterpret_cast<uint4 *>(q8 + ((long long)n * plane + pix) * a.Cp + g * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

} // namespace

static long long umma_k2(int C, long long K) // padded product count per operand kind: taps x padded channels
{
    const long long khw = C > 0 ? K / C : 0;
    return khw * ((C + 15) / 16 * 16);
}

size_t fxp_umma_workspace_bytes(int N, int C, int Hp, int Wp, int Co, long long K)
{
    const int CB = Co < 128 ? Co : 128;
    const int n_chunks = (Co + CB - 1) / CB;
    const int Cp = (C + 15) / 16 * 16;
    const long long Kp = 2 * ((umma_k2(C, K) + kSlabBytes - 1) / kSlabBytes * kSlabBytes);
    return align_up((size_t)N * Hp * Wp * Cp, 256) + align_up((size_t)n_chunks * 256 * Kp, 256) +
           align_up((size_t)Kp * 4, 256);
}

bool fxp_umma_supported(int C, int Hp, int Wp, long long K)
{
    // the offset table keeps an in-image byte offset in 30 bits
    return (long long)((C + 15) / 16 * 16) * Hp * Wp < (1LL << 30) && 2 * umma_k2(C, K) <= (1 << 20);
}

int launch_fxp_conv_umma(int N, int C, int H, int W, int ph, int pw, int Co, int KH, int KW, int OH, int OW, int sh,
                         int sw, int cap, float scale, const void *d_act, int act_dtype, const void *d_w, int w_dtype,
                         void *ws, int32_t *out, int *status, bool swizzled, cudaStream_t st)
{
    UmmaArgs a;
    const int Hp = H + 2 * ph, Wp = W + 2 * pw;
    const long long K = (long long)C * KH * KW;
    a.N = N; a.C = C; a.Hp = Hp; a.Wp = Wp; a.Co = Co; a.OH = OH; a.OW = OW; a.sh = sh; a.sw = sw;
    a.H = H; a.W = W; a.ph = ph; a.pw = pw; a.scale = scale;
    a.Cp = (C + 15) / 16 * 16;
    a.K2 = (int)umma_k2(C, K);
    a.Kp = (int)(2 * ((umma_k2(C, K) + kSlabBytes - 1) / kSlabBytes * kSlabBytes));
    a.CB = Co < 128 ? Co : 128;
    a.CBp = (a.CB + 7) / 8 * 8;
    a.CBq = (a.CBp + 31) / 32 * 32;
    a.NP = (a.CBq + a.CBp + 15) / 16 * 16;
    a.tmem_cols = 32;
    while (a.tmem_cols < 2 * a.CBq) a.tmem_cols *= 2; // the epilogue reads whole 32-column groups of both blocks
    if (a.tmem_cols > 512 || a.NP > 256) return REXSC_E_UNSUPPORTED;
    a.cap = cap;
    a.M = (long long)N * OH * OW;
    const int n_chunks = (Co + a.CB - 1) / a.CB;
    uint8_t *w8 = static_cast<uint8_t *>(ws);
    int8_t *q8 = reinterpret_cast<int8_t *>(w8);
    int8_t *wpk = reinterpret_cast<int8_t *>(w8 + align_up((size_t)N * Hp * Wp * a.Cp, 256));
    int32_t *koff = reinterpret_cast<int32_t *>(reinterpret_cast<uint8_t *>(wpk) +
                                                align_up((size_t)n_chunks * a.NP * a.Kp, 256));
    const long long n_act = (long long)N * Hp * Wp * (a.Cp / 16); // one thread per pixel and 16 channels
    const unsigned ab = (unsigned)((n_act + 255) / 256 < 148 * 16 ? (n_act + 255) / 256 : 148 * 16);
    const long long pack_items = (long long)n_chunks * a.NP * a.Kp;
    const unsigned pb = (unsigned)((pack_items + 255) / 256 < 148 * 4 ? (pack_items + 255) / 256 : 148 * 4);
    auto prep = [&](auto *x, auto *w) {
        using TA = std::remove_const_t<std::remove_pointer_t<decltype(x)>>;
        using TW = std::remove_const_t<std::remove_pointer_t<decltype(w)>>;
        fxp_umma_prep_kernel<TA, TW><<<ab + pb, 256, 0, st>>>(a, KH, KW, n_chunks, (int)ab, x, w, q8, wpk, koff);
    };
    auto prep_w = [&](auto *x) {
        switch (w_dtype) {
        case REXSC_F32: prep(x, (const float *)d_w); break;
        case REXSC_F16: prep(x, (const __half *)d_w); break;
        default: prep(x, (const __nv_bfloat16 *)d_w); break;
        }
    };
    switch (act_dtype) {
    case REXSC_F32: prep_w((const float *)d_act); break;
    case REXSC_F16: prep_w((const __half *)d_act); break;
    default: prep_w((const __nv_bfloat16 *)d_act); break;
    }
    REXSC_LAUNCH_CHECK("fxp_umma_prep_kernel");
    // Operand tiles sized by the layer: narrow layers fit more CTAs per SM, which is what hides a step's latency.  So does a
    // single weight buffer, and where there are more CTAs than SMs it hides more than the copy of the next step's weights
    // during the MMAs does (whole calls, two buffers -> one): 3x3 17 -> 497 channels, 172 CTAs: 35 -> 27 us; 5x5 33 -> 45,
    // 1319 CTAs: 123 -> 94 us; TinyConv 165 -> 155 us; with the empty blocks of its only slab left out as well, 1x1 7 -> 83
    // on 160 x 61 x 61: 228 -> 130 us (171 us with values and parity bits in one slab).  With a CTA per SM
    // and no other to hide behind the second buffer is the better one: 4x4 134 -> 78 channels, 19 CTAs: 35 against 37 us.
    const long long ctas = (a.M + kUmmaM - 1) / kUmmaM * n_chunks;
    a.w_bufs = a.Kp > 2 * kSlabBytes && ctas <= 148 ? 2 : 1;
    const size_t smem = 2 * (size_t)kUmmaM * kSlabBytes + 2 * a.w_bufs * (size_t)((a.NP + 7) / 8 * 8) * kSlabBytes + 64 + 1024;
    dim3 grid((unsigned)((a.M + kUmmaM - 1) / kUmmaM), (unsigned)n_chunks);
    auto kernel = swizzled ? fxp_conv_umma_kernel<true> : fxp_conv_umma_kernel<false>;
    REXSC_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, 128, smem, st>>>(a, q8, wpk, koff, out, status);
    REXSC_LAUNCH_CHECK("fxp_conv_umma_kernel");
    return REXSC_OK;
}

} // namespace rexsc
