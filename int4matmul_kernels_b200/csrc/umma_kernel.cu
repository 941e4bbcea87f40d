// Tensor-core path: tcgen05.mma with the dequantised weights as the A operand in tensor memory.
//
// Replaces MMA_Int4_Half (matmul_kernel.cu:219-333) and, for one or a few activation rows, MVA_Int4_Half
// (matvec_kernel.cu:198-267).  Per CTA tile: 128 weight columns (S) on the 128 tensor-memory lanes x NT
// activation rows on the MMA's N dimension, accumulated in fp32 in tensor memory over all of N (in-features).
//
//   weight producer   one thread (two, in two warps, for the weight-streaming shapes): tensor-map copies (TMA) of the
//                     packed weight rows, the keep mask and the groups' scales / zeros of one unit (128 k; 256 k for
//                     the weight-streaming shapes) into a shared-memory ring
//   activation prod.  one thread: the activation tile (NT rows x one unit of k as 128-byte-swizzled sub-tiles of 64 k);
//                     for dense int4 with up to 3 rows the whole warp, which reorders k inside the tile (see UFormat)
//   dequant warps     warpgroups of 4 warps take the units in turn; thread i of a group owns weight column i: reads
//                     its packed words from shared memory, rebuilds fp16((q - zero) * scale) in registers and
//                     writes them into its own tensor-memory lane with tcgen05.st (one packed int32 = 8 consecutive
//                     k of one column, which is exactly what a lane of the A operand holds)
//   MMA warp          one elected thread issues 8 (16) x tcgen05.mma (M = 128, N = NT, K = 16) per unit, A from tensor
//                     memory, B from the swizzled shared-memory tile, and commits to mbarriers that recycle the
//                     stages; the accumulator never leaves tensor memory until the tile is done
//   epilogue          reads the accumulator (tcgen05.ld), converts to fp16 and stores: one warpgroup of its own in the
//                     weight-streaming shapes (a CTA's last tile: from 2 rows on the dequant warpgroups as well, see last_epilogue),
//                     two warpgroups of their own (half of the columns each) in the others
//
// Configurations (Cfg<NT, PAIR, STREAM>), one CTA per SM: up to 64 rows stream the weights once from HBM - 3 dequant warpgroups, 9 (6)
// weight stages and 3 A / activation stages of 256 k, and the (tile, unit) space cut into ranges of units, one per CTA (split-K over the
// whole GPU, partial tiles summed through scratch in a fixed order).  More rows: either the same with NT = 128, units of 128 k and two
// accumulators, or NT >= 128 in whole tiles (or K parts), epilogue stores transposed through shared memory, by default launched as
// clusters of two CTAs that run each MMA together (cta_group::2, M = 256 over two SMs), see PAIR below; launch_fmt chooses.
// Every wait is bounded and reports through the status word instead of hanging.
#include "../../include/int4matmul_b200.h"

#include <cuda.h>
#include <dlfcn.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "dequant.cuh"
#include "ptx.cuh"

namespace i4mm {

namespace {


struct UmmaParams {
    OutMap om;           // where the results go (one array, or this rank's columns of several gathered arrays)
    const uint32_t* matrix;
    const uint32_t* mask;
    const __half* scales;
    const __half* zeros;
    float* partials;
    int* status;
    int rows;            // all activation rows (B * M)
    int N, S;
    int U;               // 128-k units per tile: ceil(N / 128)
    int CT;              // column tiles: ceil(S / 128)
    int MTILES;          // row tiles: ceil(rows / NT)
    int accumulate;
    int overlap;         // weight-side tensors may be read while the kernel before this one is still running
    int kparts;          // > 1: every tile's K range is cut into this many parts, one CTA (pair) each, fp32 partial outputs
                         // go to the scratch as (part, row, S) and kparts_reduce_kernel sums them (more than 64 rows only)
    GroupDiv gdiv;
    // (last: where they lay before gdiv, 128 rows on CTA pairs took 2..3 % longer in int4 and int3, 5120 x 27648 39.4 us, now 38.2)
    int whole_tiles;     // no tile is shared (weight-streaming shapes), nor K cut into parts (the others)
    unsigned int* present;   // one word per CTA, all-zero between launches (see last_epilogue)
};

// ---- formats: one 64-k part of one column -> 32 registers of fp16 pairs -----------------------------------------
// The pairs are in natural k order, except for dense int4 with PERM: there register 4r + j of packed word r holds
// (k_j, k_{j+4}) of the word's eight k, which needs no byte shuffles; the activation tile is permuted to match
// (kPermutedK: position 2j + i of every group of eight k holds k_{j + 4i}).
template <int BITS, bool SPARSE, bool PERM = false>
struct UFormat;

template <bool PERM>
struct UFormat<4, false, PERM> {
    static constexpr int WROWS = 8, MROWS = 0;       // packed rows / mask rows per 64-k part
    static constexpr bool kPermutedK = PERM;
    template <int MODE>
    __device__ static __forceinline__ void decode(uint32_t wbase, uint32_t, int half, const ColK& c, uint32_t* A, const uint32_t*) {
        if (PERM) {
            // nibbles j and j + 4 of a word sit at the same offset of its two 16-bit halves: one LOP3 per pair plants both
            // into the mantissas of (1024, 1024); the odd nibbles come out multiplied by 16
            const uint32_t off1 = hsub2_u(BASE_1_1, c.z2), off16 = hsub2_u(H2_N64, c.z2);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t w = ptx::lds32(wbase + (4 * half + r) * 512);
                const uint32_t w8 = w >> 8;
                A[4 * r + 0] = finish<4, MODE>(and_or(w, 0x000F000Fu, kMagic1024), MUL_1_1, BASE_1_1, off1, c);      // k0, k4
                A[4 * r + 1] = finish<4, MODE>(and_or(w, 0x00F000F0u, kMagic1024), H2_1_16, H2_N64, off16, c);       // k1, k5
                A[4 * r + 2] = finish<4, MODE>(and_or(w8, 0x000F000Fu, kMagic1024), MUL_1_1, BASE_1_1, off1, c);     // k2, k6
                A[4 * r + 3] = finish<4, MODE>(and_or(w8, 0x00F000F0u, kMagic1024), H2_1_16, H2_N64, off16, c);      // k3, k7
            }
            return;
        }
        const uint32_t off = hsub2_u(BASE_1_16, c.z2);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t w = ptx::lds32(wbase + (4 * half + r) * 512);
            const uint32_t y0 = prmt(w, w, 0x1010), y1 = prmt(w, w, 0x3232);   // low / high 16 bits in both lanes
            A[4 * r + 0] = finish<4, MODE>(and_or(y0, 0x00F0000Fu, kMagic1024), MUL_1_16, BASE_1_16, off, c);        // k0, k1
            A[4 * r + 1] = finish<4, MODE>(and_or(y0 >> 8, 0x00F0000Fu, kMagic1024), MUL_1_16, BASE_1_16, off, c);   // k2, k3
            A[4 * r + 2] = finish<4, MODE>(and_or(y1, 0x00F0000Fu, kMagic1024), MUL_1_16, BASE_1_16, off, c);        // k4, k5
            A[4 * r + 3] = finish<4, MODE>(and_or(y1 >> 8, 0x00F0000Fu, kMagic1024), MUL_1_16, BASE_1_16, off, c);   // k6, k7
        }
    }
};

template <bool PERM>
struct UFormat<2, false, PERM> {
    static constexpr int WROWS = 4, MROWS = 0;
    static constexpr bool kPermutedK = false;
    template <int MODE>
    __device__ static __forceinline__ void decode(uint32_t wbase, uint32_t, int half, const ColK& c, uint32_t* A, const uint32_t*) {
        const uint32_t offa = hsub2_u(BASE_1_4, c.z2), offb = hsub2_u(BASE_16_64, c.z2);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t w = ptx::lds32(wbase + (2 * half + r) * 512);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t y = h ? prmt(w, w, 0x3232) : prmt(w, w, 0x1010);   // crumbs 8h .. 8h+7 in both lanes
                const uint32_t y8 = y >> 8;
                A[8 * r + 4 * h + 0] = finish<2, MODE>(and_or(y, 0x000C0003u, kMagic1024), MUL_1_4, BASE_1_4, offa, c);
                A[8 * r + 4 * h + 1] = finish<2, MODE>(and_or(y, 0x00C00030u, kMagic1024), MUL_16_64, BASE_16_64, offb, c);
                A[8 * r + 4 * h + 2] = finish<2, MODE>(and_or(y8, 0x000C0003u, kMagic1024), MUL_1_4, BASE_1_4, offa, c);
                A[8 * r + 4 * h + 3] = finish<2, MODE>(and_or(y8, 0x00C00030u, kMagic1024), MUL_16_64, BASE_16_64, offb, c);
            }
        }
    }
};

template <bool PERM>
struct UFormat<3, false, PERM> {
    static constexpr int WROWS = 6, MROWS = 0;
    static constexpr bool kPermutedK = false;
    template <int MODE>
    __device__ static __forceinline__ void decode(uint32_t wbase, uint32_t, int blk, const ColK& c, uint32_t* A, const uint32_t*) {
        const uint32_t off = hsub2_u(BASE_1_8, c.z2);
        const uint32_t w0 = ptx::lds32(wbase + (3 * blk) * 512), w1 = ptx::lds32(wbase + (3 * blk + 1) * 512), w2 = ptx::lds32(wbase + (3 * blk + 2) * 512);
        // the 96-bit stream in 12-bit chunks: chunk j holds fields 4j .. 4j+3 = pairs (2j, 2j+1)
        uint32_t ch[8];
        ch[0] = w0;
        ch[1] = w0 >> 12;
        ch[2] = __funnelshift_r(w0, w1, 24);
        ch[3] = w1 >> 4;
        ch[4] = w1 >> 16;
        ch[5] = __funnelshift_r(w1, w2, 28);
        ch[6] = w2 >> 8;
        ch[7] = w2 >> 20;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t y = prmt(ch[j], ch[j], 0x1010);
            A[2 * j + 0] = finish<3, MODE>(and_or(y, 0x00380007u, kMagic1024), MUL_1_8, BASE_1_8, off, c);
            A[2 * j + 1] = finish<3, MODE>(and_or(y >> 6, 0x00380007u, kMagic1024), MUL_1_8, BASE_1_8, off, c);
        }
    }
};

template <bool PERM>
struct UFormat<4, true, PERM> {
    static constexpr int WROWS = 4, MROWS = 2;
    static constexpr bool kPermutedK = false;
    template <int MODE>
    __device__ static __forceinline__ void decode(uint32_t wbase, uint32_t mbase, int blk, const ColK& c, uint32_t* A, const uint32_t* lut) {
        // a 32-block of this column: the 64-bit word of its 16 kept nibbles (in increasing k) and its keep-mask
        uint32_t lo = ptx::lds32(wbase + (2 * blk) * 512), hi = ptx::lds32(wbase + (2 * blk + 1) * 512);
        const uint32_t m = ptx::lds32(mbase + blk * 512);
#pragma unroll
        for (int step = 0; step < 4; ++step) {               // 8 positions each
            uint32_t pairs[4];
            sparse_expand<MODE>(lo, hi, m, step, lut, c, pairs);
#pragma unroll
            for (int i = 0; i < 4; ++i) A[4 * step + i] = pairs[i];
        }
    }
};

template <class F, int MODE>
__device__ __forceinline__ void decode_part(uint32_t wbase, uint32_t mbase, const ColK& c, uint32_t (&A)[32], const uint32_t* lut) {
#pragma unroll
    for (int half = 0; half < 2; ++half) F::template decode<MODE>(wbase, mbase, half, c, A + 16 * half, lut);
}

// Bits that are set where a column's group is not in the fast mode, for two groups at once: s, z their scales and zero-points, zi = z + 1024;
// BOUND + the fp16 bits of the largest zero-point = 0x7FFF
template <uint32_t BOUND>
__device__ __forceinline__ uint32_t not_fast_bits(uint32_t s, uint32_t z, uint32_t zi) {
    return ((z | s | ((z & 0x7FFF7FFFu) + BOUND * 0x10001u)) & 0x80008000u) | (hadd2_u(zi, H2_N1024) ^ z);
}

template <class F, int H>
struct WStage {     // one stage of the packed-weight ring: one unit = H parts of 64 k
    static constexpr int kW = 0;                                 // H * WROWS packed rows of 512 B
    static constexpr int kMask = H * F::WROWS * 512;             // H * MROWS mask rows of 512 B
    static constexpr int kS = kMask + H * F::MROWS * 512;        // H rows of scales (groups g0 .. g0 + H - 1), 256 B each
    static constexpr int kZ = kS + H * 256;                      // H rows of zeros
    static constexpr int kBytes = kZ + H * 256;
};

constexpr int kMaxWStages = 16;
constexpr int kMaxABStages = 6;

// The fast mode takes zero-points up to 512 (16:32, whose expansion XORs them into the nibbles: up to 127): kFastBound + the fp16 bits of
// the largest one = 0x7FFF.
template <bool SPARSE>
constexpr uint32_t kFastBound = SPARSE ? 0x280Fu : 0x1FFFu;
constexpr uint32_t kWideBound = 0x2407u;          // MODE_WIDE: up to 255

template <int NT, bool PAIR, bool STREAM = NT <= 64>
struct Cfg {
    // packed-weight ring (128 k per stage).  Few rows: the kernel streams weights from HBM, and the ring has to
    // cover the DRAM latency; many rows: weights are a trickle next to the activation tiles
    // Weight-streaming shapes: everything doubled, K split over the CTAs with a scratch reduction, an epilogue from registers that the MMA warp
    // wakes (named barrier): all of up to 64 rows, and NT = 128 where launch_fmt takes it.  The others: whole tiles, or K parts (choose_kparts),
    // and epilogue stores that go through a shared-memory transposition tile.  (33..64 rows in whole tiles of 64 rows, two CTAs an SM, or K parts:
    // 48 rows 13824 x 5120 int4 26.6 us, now 17.4, 16:32 37.8 / 20.8; 5120 x 20480 57.1 / 23.0, 54.9 / 29.3; 1024 x 1024 8.9 / 6.5, 9.6 / 7.6.)
    static constexpr bool kStream = STREAM;
    // NT = 128..192: an MMA of N <= 192 takes 512..768 cycles per 128 k, the dequantisation of its weights with two
    // warpgroups ~1400, so these shapes get four warpgroups as well, and a deeper weight ring
    // (single CTAs have the shared memory for the 4 A / activation stages that four warpgroups need only at NT = 128)
    static constexpr bool kDequantBound = !STREAM && (NT == 128 || (PAIR && NT >= 128 && NT <= 192));
    // A stage of either ring is waited for by parity, which tells a completed phase only from the one before it.
    // Where the weight stages are not a multiple of the warpgroups, consecutive uses of a stage belong to different
    // warpgroups, and one could poll for a stage's next fill while the previous one, meant for another warpgroup, has
    // not landed yet (tensor-map copies may complete out of order) and take the stale phase for its own: there the
    // dequant warps first wait, like the producer, until the previous use has been released (kWGuard).  And there
    // are at least as many A stages as warpgroups (checked in the kernel).
    // A unit (one stage of every ring) is kHalves parts of 64 k.  The producers and the MMA issuer are single threads
    // whose loops cost ~500 cycles per stage whatever its size (an mbarrier wait ~190 cycles even when it is already
    // complete, expect_tx + the copy's issue another ~190): at 128 k per stage that alone is ~27 us for 16384 x 16384
    // weights on 148 SMs, so the weight-streaming shapes use 256-k units (but NT = 128: 128 k, its activation stages would not fit).
    static constexpr int kHalves = NT <= 64 ? 4 : 2;
    static constexpr int kWStages = kStream ? (NT <= 16 || NT == 128 ? 9 : 6) : kDequantBound ? 6 : 3;
    // staging slots (units of look-ahead) for activation rows that are reordered on their way into the A / activation
    // stages (umma_kernel's PERM)
    static constexpr int kXStaging = 4;
    static constexpr int kWG = kStream ? 3 : kDequantBound ? 4 : 2;   // dequant warpgroups (4 warps each), taking units in turn
    static constexpr int kABStages = NT == 128 ? 4 : 3;   // ring of (A in tensor memory, activation tile in shared memory) pairs, one unit per stage
    static constexpr bool kWGuard = kWStages % kWG != 0;
    // many rows: two epilogue warpgroups, each draining half of the accumulator's columns, so that the next tile's
    // MMAs wait half as long for the accumulator
    static constexpr int kEpiGroups = kStream ? 1 : 2;
    // The weight-streaming shapes have two weight-producer threads (in two warps) that fill the stages in turn: one
    // thread's loop (wait ~190 cycles, expect_tx + copies ~250) delivers a 16 KB stage per ~500-700 cycles, about
    // 4-5 TB/s over the whole GPU, which is less than the memory system can stream.
    static constexpr int kWProducers = kStream ? 2 : 1;
    static constexpr int kWarps = 4 * kWG + 4 * kEpiGroups + 3 + (kWProducers - 1);  // + weight producer(s), activation producer, MMA issuer
    static constexpr int kThreads = kWarps * 32;
    static constexpr int kDCols = NT < 32 ? 32 : NT;                  // accumulator columns
    static constexpr int kDBufs = kStream && NT == 128 ? 2 : 1;       // accumulators, used by the tiles in turn
    static constexpr int kACol0 = kDBufs * kDCols;                             // A stages follow: 32 columns per 64 k
    static constexpr int kAStageCols = 32 * kHalves;
    static constexpr int kColsUsed = kACol0 + kAStageCols * kABStages;
    static constexpr int kTmemCols = kColsUsed <= 256 ? 256 : 512;
    static constexpr int kSlotVecs = NT / 4 * 128;                    // one CTA's partial tile in the scratch: [4 rows][128 columns] of 16 bytes
    static constexpr int kSlots = NT <= 32 ? 1 : 2;                   // of those per CTA, see last_epilogue
};

// A / activation stages.  A CTA of a pair holds only half of each activation tile, which leaves shared memory for as
// many stages as tensor memory has columns for (accumulator + 64 per stage <= 512).
template <int NT, bool PAIR, bool STREAM>
struct ABStages {
    static constexpr int value = !PAIR ? Cfg<NT, false, STREAM>::kABStages : (Cfg<NT, true>::kDCols + 64 * 5 <= 512 ? 5 : 4);   // pairs: 128-k units
};

struct Barriers {
    unsigned long long w_full[kMaxWStages], w_empty[kMaxWStages];
    unsigned long long ab_full[kMaxABStages];  // 4 dequant warps + the activation producer (with its transaction bytes)
    unsigned long long ab_free[kMaxABStages];  // tcgen05.commit: the MMAs that read the stage are done
    unsigned long long d_full, d_empty[2];     // d_empty: one per accumulator
};

struct TensorMaps {
    CUtensorMap x;   // fp16 (rows, N):        box 64 k x NT rows, 128-byte swizzle; weight-streaming shapes: seen as
                     //                        (N / 64, rows, 64) with box kHalves x NT x 64, one copy per unit
    CUtensorMap w;   // int32 (R, S):          box 128 columns x kHalves * WROWS rows
    CUtensorMap m;   // int32 (N / 32, S):     box 128 columns x kHalves * MROWS rows (sparse format only)
    CUtensorMap s;   // fp16 (n_groups, S):    box 128 columns x kHalves rows
    CUtensorMap z;
};

// Rows 0 .. n - 1 of one column to every destination (out0: the first row in the first one).  The first destination's stores are
// predicated, without the branch and the loop over destinations per row (5120 x 20480 int4, 32 rows: 24.9 -> 23.5 us).  (Rows and columns changing
// places among eight lanes, so that a store is 16 bytes, was no faster: 72 rows 2048 x 16384 int4 13.2 / 13.1 us, but 16 rows 9.8 / 10.2.)
template <int RB>
__device__ __forceinline__ void store_rows(const OutMap& om, __half* out0, long long ld, int n_dst, const __half (&h)[RB], int n) {
#pragma unroll
    for (int i = 0; i < RB; ++i)
        if (i < n) out0[(size_t)i * ld] = h[i];
    for (int d = 1; d < n_dst; ++d) {
        __half* const out = om.dst[d] + (out0 - om.dst[0]);
#pragma unroll
        for (int i = 0; i < RB; ++i)
            if (i < n) out[(size_t)i * ld] = h[i];
    }
}

// The epilogue of the weight-streaming shapes.  Split-K: the CTAs b_lo .. b_hi share a tile.  b_lo,
// which owns its first units and reaches them last, adds the others' partial tiles to its own accumulator in CTA order - a fixed
// order, so results are reproducible.  A partial sum is a 32-bit word that is never zero (share_word), four rows of
// a column in one 16-byte store, so no fence, counter or second round trip is needed: a reader knows each word by itself, and clears
// what it has read, which leaves the scratch all-zero for the next launch.  A CTA has at most one
// tile that it shares and goes on from, before its last one, so there are two functions.
// CTAs are numbered against the order in which blocks start (CTA b is block G - 1 - b), so b_lo waits only for blocks that started before it:
// a launch gets through on however few SMs other streams leave it (with b_lo's block starting first, two were needed).  For the waits of more
// than 32 rows see last_epilogue.
// What a thread waits for are its loads, so fewer and wider ones count: with one 64-bit word (value | tag) per row, int4 16 rows 20480 x 5120
// 22.3 us, now 19.7; 5120 x 5120 13.2 / 10.2; 16384 x 2048 17.0 / 12.4; 32 rows 25.1 / 21.1, 15.6 / 11.7, 20.4 / 14.9; one row 18.4 / 17.7, 10.3 / 9.7,
// 12.7 / 11.5.
__device__ __forceinline__ uint32_t share_word(uint32_t v) { return __float_as_uint(__uint_as_float(v) + 0.0f) ^ 0x80000000u; }   // (-0 goes as +0)
__device__ __forceinline__ float share_value(uint32_t w) { return __uint_as_float(w ^ 0x80000000u); }

// A tile before a CTA's last one, by the epilogue warps: a whole tile, or (share: this lane's column of the CTA's slot) the CTA's share
// of a tile that another CTA sums.  The next tile's MMAs wait for it.  Not inlined and with its arguments by value: with `p` by
// reference a call cost ~1 us (1024 x 32768 int4, 5 rows, two or three tiles a CTA: 16.2 us, now 12.9), and inlined it slowed the
// decode loop (13824 x 5120 int4, 4 rows: 17.4 us, now 16.5).
// out0: the column's first output; rows / out_rows: rows of the launch, and those that this lane stores.
template <int NT>
__device__ __noinline__ bool early_epilogue(const OutMap& om, int n_dst, long long ld, __half* out0, int rows, int out_rows, int accumulate,
                                            uint4* share, uint32_t acc, uint32_t bar_id, uint32_t d_empty, uint32_t s_abort) {
    const uint32_t lane_addr = acc + ((threadIdx.x & 96u) << 16);
    auto release = [&]() {
        ptx::tc_fence_before_sync();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(d_empty);
    };
    __half old[8];
    auto load_old = [&](int rb) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            old[i] = __ushort_as_half(0);
            if (accumulate && rb + i < out_rows) old[i] = out0[(size_t)(rb + i) * ld];
        }
    };
    if (!share) load_old(0);
    ptx::named_bar_sync(bar_id, 128 + 32);         // released by the MMA warp once the accumulator is complete
    if (ptx::lds32(s_abort)) return false;
    ptx::tc_fence_after_sync();
    if (share) {
#pragma unroll 1
        for (int rb = 0; rb < rows; rb += 16) {
            uint32_t v[16];
            ptx::tmem_ld16(lane_addr + rb, v);
            ptx::tc_wait_ld();
            if (rb + 16 >= rows) release();
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                if (rb + i < rows)
                    ptx::st_relaxed_gpu_v4(share + (rb + i) / 4 * 128, make_uint4(share_word(v[i]), share_word(v[i + 1]), share_word(v[i + 2]), share_word(v[i + 3])));
        }
        return true;
    }
    if (NT == 64 && !accumulate) {
        // converted and held in registers, so that the accumulator is free before the stores
        uint32_t h2[NT / 2];
#pragma unroll
        for (int rb = 0; rb < NT; rb += 16) {
            uint32_t v[16];
            ptx::tmem_ld16(lane_addr + rb, v);
            ptx::tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2)
                h2[(rb + i) / 2] = h2_as_u32(__floats2half2_rn(__uint_as_float(v[i]), __uint_as_float(v[i + 1])));
        }
        release();
#pragma unroll
        for (int rb = 0; rb < NT; rb += 16) {
            __half h[16];
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                h[i] = __low2half(u32_as_h2(h2[(rb + i) / 2]));
                h[i + 1] = __high2half(u32_as_h2(h2[(rb + i) / 2]));
            }
            store_rows<16>(om, out0 + (size_t)rb * ld, ld, n_dst, h, out_rows - rb);
        }
        if (n_dst > 1) __threadfence_system();
        return true;
    }
    auto finish_rows = [&](auto rb_tag, int rb) {
        constexpr int RB = decltype(rb_tag)::value;
        uint32_t v[RB];
        ptx::tmem_ld(lane_addr + rb, v);
        ptx::tc_wait_ld();
        if (rb + RB >= rows) release();
        __half h[RB];
#pragma unroll
        for (int i = 0; i < RB; ++i) {
            const float f = __uint_as_float(v[i]);
            h[i] = __float2half_rn(accumulate ? f + __half2float(old[i]) : f);
        }
        store_rows<RB>(om, out0 + (size_t)rb * ld, ld, n_dst, h, out_rows - rb);
    };
    if (rows <= 4) {
        finish_rows(std::integral_constant<int, 4>(), 0);
    } else {
#pragma unroll 1
        for (int rb = 0; rb < rows; rb += 8) {
            if (rb > 0) load_old(rb);
            finish_rows(std::integral_constant<int, 8>(), rb);
        }
    }
    if (n_dst > 1) __threadfence_system();         // as in umma_kernel's epilogue
    return true;
}

// Adds the shares of n partners, PB at a time, to the sums of NG groups of four rows (the first `here` of them are there) and clears them.
// at(k, j): partner k's words of group j.  NG x PB loads are in flight, and everything that is missing is asked for again at once: word by word
// each would cost a round trip of its own.
constexpr uint32_t kShareSpins = 1u << 22;        // seconds: a poll is a round trip to L2
template <int NG, int PB, class At>
__device__ __forceinline__ void add_shares(float (&sum)[4 * NG], int n, int here, int* status, bool& waiting_ok, At at) {
#pragma unroll 1
    for (int q = 0; q < n; q += PB) {
        uint4 w[PB][NG];
        auto missing = [&](int k, int j) -> bool {
            return q + k < n && j < here && (w[k][j].x == 0u || w[k][j].y == 0u || w[k][j].z == 0u || w[k][j].w == 0u);
        };
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
            for (int j = 0; j < NG; ++j) w[k][j] = make_uint4(0, 0, 0, 0);
        for (uint32_t spins = 0; waiting_ok; ++spins) {
#pragma unroll
            for (int k = 0; k < PB; ++k)
#pragma unroll
                for (int j = 0; j < NG; ++j)
                    if (missing(k, j)) w[k][j] = ptx::ld_relaxed_gpu_v4(at(q + k, j));
            bool any = false;
#pragma unroll
            for (int k = 0; k < PB; ++k)
#pragma unroll
                for (int j = 0; j < NG; ++j) any |= missing(k, j);
            if (!any) break;
            if (spins >= kShareSpins) {                        // a contributor never delivered: report, stop waiting
                atomicExch(status, 34);
                waiting_ok = false;
            }
            __nanosleep(20);
        }
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
            for (int j = 0; j < NG; ++j)
                if (q + k < n && j < here) {
                    const uint4 x = w[k][j];
                    sum[4 * j] += share_value(x.x);
                    sum[4 * j + 1] += share_value(x.y);
                    sum[4 * j + 2] += share_value(x.z);
                    sum[4 * j + 3] += share_value(x.w);
                    ptx::st_relaxed_gpu_v4(at(q + k, j), make_uint4(0, 0, 0, 0));
                }
    }
}

// The CTAs that share a tile, and how many of them, from b_lo on, sum it
struct TileCtas {
    int b_lo, b_hi, members;
    __device__ __forceinline__ int first_group(int groups, int member) const { return (groups * member + members - 1) / members; }
};
constexpr int kLeftWords = 10;                    // (see the assertion in launch_nt)
constexpr uint32_t kLeaveSpins = 1u << 7;         // ~0.15 ms, far more than the starts of CTAs that do run side by side differ
// CTA bb's slot, for up to 32 rows one, else two: its share of the tile that it shares and goes on from, and the one of its last tile
template <int NT>
__device__ __forceinline__ uint4* share_slot(uint4* slots, const TileCtas& ctas, int bb) {
    return slots + (size_t)(NT > 32 ? 2 * bb + (bb < ctas.b_lo + ctas.members ? 1 : 0) : bb) * Cfg<NT, false, true>::kSlotVecs;
}

// The groups of member `r`, which left them to b_lo (see last_epilogue), this part of them: its own share is in its slot; the same sums in the same order.
template <int NT>
__device__ __noinline__ bool finish_for(const UmmaParams& p, __half* out, bool col_ok, int rows, uint4* slots, TileCtas ctas, int r, int part, int parts) {
    bool waiting_ok = true;
    const int groups = (rows + 3) / 4, lo = ctas.first_group(groups, r), n_groups = ctas.first_group(groups, r + 1) - lo, g_end = lo + n_groups * (part + 1) / parts;
    const int who = ctas.b_lo + r;
#pragma unroll 1
    for (int g = lo + n_groups * part / parts; g < g_end; ++g) {
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, own[4] = {0.f, 0.f, 0.f, 0.f};
        add_shares<1, 1>(sum, ctas.b_hi - ctas.b_lo, 1, p.status, waiting_ok,
                         [&](int k, int) { return share_slot<NT>(slots, ctas, ctas.b_lo + k + (k >= r ? 1 : 0)) + g * 128; });
        add_shares<1, 1>(own, 1, 1, p.status, waiting_ok, [&](int, int) { return share_slot<NT>(slots, ctas, who) + g * 128; });
        __half* const out0 = out + (size_t)(4 * g) * p.om.ld;
        const int n = col_ok ? min(4, rows - 4 * g) : 0;
        __half h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float f = own[i] + sum[i];
            if (p.accumulate && i < n) f += __half2float(out0[(size_t)i * p.om.ld]);
            h[i] = __float2half_rn(f);
        }
        store_rows<4>(p.om, out0, p.om.ld, p.om.n_dst, h, n);
    }
    return waiting_ok;
}

// A CTA's last tile: units t0 .. t0 + units - 1.  What bounds it is the number of dependent round trips to L2 (~0.7 us each) and the words a
// CTA reads between the last MMA and the end of the launch, so the tile can be left to all of the CTA's warpgroups (the dequant warps
// have nothing else to do by then), `part` of `parts` of its groups of four rows each.  (When: see spread_last.)
// Up to 32 rows b_lo sums the tile, with 4 partners' words a thread in flight.  More rows are too many words for one CTA (128 rows
// 5120 x 5120 int4: the sum took 14 of the launch's 34 K cycles on 40 of the GPU's SMs, now 6 K): there all CTAs whose last tile it is - all that
// share it but one that goes on to the next tile, whose share came early - sum some groups each; a CTA writes its sums of the others'
// groups and adds theirs to its own.  (us, b_lo alone / all: int4 48 rows 13824 x 5120 18.3 / 17.3, 128 rows 26.2 / 22.0, 5120 x 5120
// 19.4 / 15.6; but 16 rows 2048 x 8192 8.7 / 9.3, 5120 x 6976 11.3 / 11.9.)
// A member but b_lo so needs shares of blocks that start after it, and must not keep its SM from them.  b_lo's block starts last of all, and then
// writes 1 into the `present` word of each member.  A member that does not find it within kLeaveSpins writes 2 and leaves: the share of its own
// groups goes into its slot as well, and b_lo, which finds the 2, sums them in its place (finish_for).  Beside each other the CTAs of a tile have
// settled this long before the last MMA; s_left says what was settled: a member's word 0 whether it leaves, b_lo's bits who has left.
// bar_id, bar_threads: the named barrier at which the MMA warp says that the accumulator is complete (once per call, also where this
// part has no rows).  Inlined: a call cost ~1 us here as well.
template <int NT>
__device__ __forceinline__ bool last_epilogue(const OutMap& om, int n_dst, long long ld, __half* out, bool col_ok, int rows, int accumulate, uint4* slots, int* status,
                                           TileCtas ctas, const UmmaParams& p, const volatile uint32_t* s_left, uint32_t acc, int part, int parts, uint32_t bar_id, uint32_t bar_threads, uint32_t s_abort) {
    constexpr bool kAll = NT > 32;                             // every CTA whose last tile it is sums some groups
    const int b_lo = ctas.b_lo, b_hi = ctas.b_hi, members = ctas.members, me = (int)(gridDim.x - 1 - blockIdx.x), groups = (rows + 3) / 4;
    auto slot_of = [&](int bb) { return share_slot<NT>(slots, ctas, bb); };
    auto wait_accumulator = [&]() -> bool {
        __syncwarp();
        ptx::named_bar_sync(bar_id, bar_threads);      // released by the MMA warp once the accumulator is complete
        if (ptx::lds32(s_abort)) return false;
        ptx::tc_fence_after_sync();
        return true;
    };
    auto share_group = [&](const uint32_t* v) { return make_uint4(share_word(v[0]), share_word(v[1]), share_word(v[2]), share_word(v[3])); };
    bool waiting_ok = true;
    // groups g .. g + NG - 1 up to g_end: partners' shares + accumulator + old outputs -> outputs
    auto finish = [&](auto ng_tag, auto pb_tag, int g, int g_end, bool& ready) -> bool {
        constexpr int NG = decltype(ng_tag)::value, PB = decltype(pb_tag)::value;
        const int here = g_end - g, n = min(4 * here, rows - 4 * g);
        __half* const out0 = out + (size_t)(4 * g) * ld;
        float sum[4 * NG];
        __half old[4 * NG];
#pragma unroll
        for (int i = 0; i < 4 * NG; ++i) {
            sum[i] = 0.f;
            old[i] = __ushort_as_half(0);
            if (accumulate && i < n && col_ok) old[i] = out0[(size_t)i * ld];
        }
        // (b_lo .. b_hi without this CTA)
        add_shares<NG, PB>(sum, b_hi - b_lo, here, status, waiting_ok,
                           [&](int k, int j) { return slot_of(b_lo + k + (!kAll || b_lo + k >= me ? 1 : 0)) + (g + j) * 128; });
        if (!ready && !wait_accumulator()) return false;
        ready = true;
        __half h[4 * NG];
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            uint32_t v[4] = {0u, 0u, 0u, 0u};
            if (j < here) {
                ptx::tmem_ld4(acc + 4 * (g + j), v);
                ptx::tc_wait_ld();
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float f = __uint_as_float(v[i]) + sum[4 * j + i];
                if (accumulate) f += __half2float(old[4 * j + i]);
                h[4 * j + i] = __float2half_rn(f);
            }
        }
        store_rows<4 * NG>(om, out0, ld, n_dst, h, col_ok ? n : 0);
        return true;
    };
    using std::integral_constant;
    if constexpr (!kAll) {
        const int g = groups * part / parts, g_end = groups * (part + 1) / parts;
        if (me != b_lo) {
            if (!wait_accumulator()) return false;
#pragma unroll
            for (int j = 0; j < 2; ++j)                        // (NT / 16 groups a part, 2 where the epilogue warps have up to 6 rows)
                if (g + j < g_end) {
                    uint32_t v[4];
                    ptx::tmem_ld4(acc + 4 * (g + j), v);
                    ptx::tc_wait_ld();
                    ptx::st_relaxed_gpu_v4(slot_of(me) + (g + j) * 128, share_group(v));
                }
            return true;
        }
        bool ready = false;
        if (g_end - g <= 1) {
            if (!finish(integral_constant<int, 1>(), integral_constant<int, 4>(), g, g_end, ready)) return false;
        } else {
            if (!finish(integral_constant<int, 2>(), integral_constant<int, 4>(), g, g_end, ready)) return false;
        }
    } else {
        // this CTA's groups [lo, hi); of those, this part's
        const int rank = me - b_lo, lo = ctas.first_group(groups, rank), hi = ctas.first_group(groups, rank + 1);
        const int g_end = lo + (hi - lo) * (part + 1) / parts;
        int g = lo + (hi - lo) * part / parts;
        bool ready = false;
        if (members > 1) {
            if (!wait_accumulator()) return false;
            ready = true;
            const bool leave = rank > 0 && s_left[0] != 0u;
            const int end = groups * (part + 1) / parts;
#pragma unroll 1
            for (int j = groups * part / parts; j < end; j += 2) {
                uint32_t v[8];
                ptx::tmem_ld8(acc + 4 * j, v);
                ptx::tc_wait_ld();
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (j + k < end && (leave || j + k < lo || j + k >= hi)) ptx::st_relaxed_gpu_v4(slot_of(me) + (j + k) * 128, share_group(v + 4 * k));
            }
            if (leave) return true;
        }
        // (once at least: every part meets the MMA warp)
        if (b_hi - b_lo <= 2) {
            do {
                if (!finish(integral_constant<int, 4>(), integral_constant<int, 2>(), g, g_end, ready)) return false;
            } while ((g += 4) < g_end);
        } else {
            do {
                if (!finish(integral_constant<int, 2>(), integral_constant<int, 4>(), g, g_end, ready)) return false;
            } while ((g += 2) < g_end);
        }
        if (rank == 0 && members > 1) {                // (s_left is written then)
#pragma unroll 1
            for (int r0 = 0; r0 < members; r0 += 32)
#pragma unroll 1
                for (uint32_t left = s_left[r0 / 32]; left != 0u && waiting_ok; left &= left - 1u)
                    waiting_ok = finish_for<NT>(p, out, col_ok, rows, slots, ctas, r0 + __ffs((int)left) - 1, part, parts);
        }
    }
    if (n_dst > 1) __threadfence_system();                // as in umma_kernel's epilogue
    return true;
}

// The same as a call of its own.  Which form an instance takes is a matter of the decode loop's registers: up to 32 rows it is faster without the
// inlined form beside it (us, inlined / called: one row 16384 x 16384 16:32 52.7 / 50.5, int3 39.4 / 38.6, 16 rows int4 38.6 / 37.8), but with the
// permuted k order (one row int4 35.5 / 37.0) and more rows, whose call keeps more registers (48 rows 5120 x 6976 int4 13.3 / 15.5).
template <int NT>
__device__ __noinline__ bool last_epilogue_call(const OutMap& om, int n_dst, long long ld, __half* out, bool col_ok, int rows, int accumulate, uint4* slots, int* status,
                                                TileCtas ctas, const UmmaParams& p, const volatile uint32_t* s_left, uint32_t acc, int part, int parts, uint32_t bar_id, uint32_t bar_threads, uint32_t s_abort) {
    return last_epilogue<NT>(om, n_dst, ld, out, col_ok, rows, accumulate, slots, status, ctas, p, s_left, acc, part, parts, bar_id, bar_threads, s_abort);
}

// PAIR: launched as clusters of two CTAs (two SMs) that run every MMA together (cta_group::2, M = 256): the pair's
// tile is 256 weight columns x NT rows, each CTA dequantises its own 128 columns and loads only half of the rows of
// the activation tile, which halves the L2 -> shared-memory traffic that bounds the many-row shapes.
// PERM (up to 3 rows of dense int4 only): the cheaper k order of UFormat, with the activations reordered to match.
template <int BITS, bool SPARSE, int NT, bool PAIR, bool PERM = false, bool STREAM = NT <= 64>
__global__ void __launch_bounds__(Cfg<NT, PAIR, STREAM>::kThreads, 1)
umma_kernel(const __grid_constant__ TensorMaps tm, const __grid_constant__ UmmaParams p, const __half* x) {
    using C = Cfg<NT, PAIR, STREAM>;
    using F = UFormat<BITS, SPARSE, PERM>;
    static_assert(!PERM || (C::kStream && F::kPermutedK), "the permuted k order is for dense int4 weight streaming");
    constexpr int H = C::kHalves;                                    // 64-k parts per unit
    using WS = WStage<F, H>;
    static_assert(!PAIR || (NT >= 128 && !C::kStream), "CTA pairs are for the many-row shapes");
    static_assert((2 * C::kWStages) % C::kWG == 0, "every second use of a weight stage must be by the same warpgroup");
    static_assert(ABStages<NT, PAIR, STREAM>::value >= C::kWG, "fewer A stages than warpgroups: a parity wait could see the phase before last");
    constexpr int kBHalfBytes = (PAIR ? NT / 2 : NT) * 128;        // one 64-k activation sub-tile held by this CTA
    constexpr int kBStageBytes = H * kBHalfBytes;
    // single CTAs at NT = 256 have no shared memory left for a second transposition tile: the second epilogue group idles
    constexpr int kEpiGroups = (C::kEpiGroups == 2 && (PAIR || NT < 256)) ? 2 : 1;
    constexpr int kEpiWarp0 = 4 * C::kWG;                           // first epilogue warp (a multiple of 4: lane quarter = warp % 4)
    constexpr int kWProducer = kEpiWarp0 + 4 * C::kEpiGroups, kBProducer = kWProducer + 1, kMma = kWProducer + 2;
    constexpr int kWProducer2 = kWProducer + 3;                     // only when Cfg::kWProducers == 2
    constexpr int kABStages = ABStages<NT, PAIR, STREAM>::value;
    extern __shared__ __align__(1024) unsigned char smem[];      // [B ring (1024-aligned tiles)][W ring]
    __shared__ __align__(8) Barriers bars;
    __shared__ uint32_t lut[SPARSE ? kSparseLutEntries : 1];
    __shared__ uint32_t tmem_base_smem;
    __shared__ struct { TileCtas ctas; int ct, mt; uint32_t buf; } s_last;      // (weight-streaming shapes)
    __shared__ volatile uint32_t s_left[C::kStream && NT > 32 ? kLeftWords : 1];
    __shared__ volatile int s_abort;     // set by a warp that gives up on the accumulator (the MMA warp before it releases the epilogue
                                         // warps for the last time; an epilogue warp before its group's next named barrier)

    // the shuffle tells the compiler that the warp index is warp-uniform: role dispatch, stage indices and barrier
    // addresses derived from it then live in uniform registers instead of costing vector-ALU instructions
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
    const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;       // in the pair; rank 0 leads (issues the MMAs, owns the pair's barriers)
    const uint32_t smem0 = (ptx::smem_u32(smem) + 1023u) & ~1023u;
    const uint32_t b_ring = smem0;
    const uint32_t w_ring = smem0 + kABStages * kBStageBytes;
    const uint32_t epi_tile = w_ring + C::kWStages * WS::kBytes;     // 4 KB transposition tile per epilogue warpgroup (NT >= 128)
    const uint32_t x_staging = epi_tile;                             // weight-streaming shapes (no transposition tile): activation staging ring

    // ---- set-up, spread over warps so that nothing waits for one thread ----
    // The weight producer's warp initialises the weight ring's barriers itself and does not wait for the rest of the
    // CTA (it only arrives on the set-up barrier): its first copies are in flight while tensor memory is allocated.
    if (warp == kWProducer) {
        if (lane == 0) {
            ptx::prefetch_tmap(&tm.w);
            if (SPARSE) ptx::prefetch_tmap(&tm.m);
        }
        if (lane < C::kWStages) {
            ptx::mbar_init(ptx::smem_u32(&bars.w_full[lane]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars.w_empty[lane]), 4);
        }
        ptx::fence_mbar_init();
        __syncwarp();
        if (PAIR) ptx::cluster_sync_all();        // the other CTA arrives on this one's barriers: both must be set up first
        else ptx::named_bar_arrive(3, C::kThreads);
    } else {
        if (warp == 0) {
            if (lane < kABStages) {
                // a pair's stage is full when the dequant warps of both CTAs and both activation halves have arrived
                ptx::mbar_init(ptx::smem_u32(&bars.ab_full[lane]), PAIR ? 4 + 4 + 1 : 4 + 1);
                ptx::mbar_init(ptx::smem_u32(&bars.ab_free[lane]), 1);
            }
            if (lane == 31) {
                ptx::mbar_init(ptx::smem_u32(&bars.d_full), 1);
                ptx::mbar_init(ptx::smem_u32(&bars.d_empty[0]), (PAIR ? 8 : 4) * kEpiGroups);
                ptx::mbar_init(ptx::smem_u32(&bars.d_empty[1]), 4);
                s_abort = 0;
            }
            ptx::fence_mbar_init();
        }
        if (SPARSE && warp < 8) lut[warp * 32 + lane] = sparse_selectors(warp * 32 + lane);   // (warps 0..7 are dequant warps in every configuration)
        if (warp == kMma) {
            if (PAIR) {
                ptx::tmem_alloc_pair(ptx::smem_u32(&tmem_base_smem), C::kTmemCols);
                ptx::tmem_relinquish_pair();
            } else {
                ptx::tmem_alloc(ptx::smem_u32(&tmem_base_smem), C::kTmemCols);
                ptx::tmem_relinquish();
            }
        }
        if (warp == kBProducer && lane == 0) {
            ptx::prefetch_tmap(&tm.x);
            ptx::prefetch_tmap(&tm.s);
            ptx::prefetch_tmap(&tm.z);
        }
        ptx::tc_fence_before_sync();
        if (PAIR) ptx::cluster_sync_all();
        else ptx::named_bar_sync(3, C::kThreads);
        ptx::tc_fence_after_sync();
    }
    const uint32_t tmem_base = tmem_base_smem;       // not valid in the weight producer's warp, which never uses it

    // ---- this CTA's share of the (tile, unit) space; one unit = H x 64 k.  Whole tiles unless the split-K variant ----
    const long long U = p.U;
    const int CTd = PAIR ? (p.CT + 1) / 2 : p.CT;                  // column tiles of a CTA, or column-tile pairs of a CTA pair
    const long long n_tiles = (long long)p.MTILES * CTd;
    // (weight-streaming shapes: numbered against the order in which blocks start, see early_epilogue)
    const long long G = PAIR ? gridDim.x / 2 : gridDim.x, b = PAIR ? blockIdx.x / 2 : C::kStream ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    // tile index -> this CTA's column tile (may lie past the last one in a pair: loads are zero-filled, stores masked) and row tile
    // Column tiles vary fastest.  (Row tiles fastest would read each packed-weight tile from HBM only once, but then every
    // SM asks L2 for the same activation lines at the same moment, and that hot spot cost 3-25 % when measured.)
    auto tile_ct = [&](long long tile) -> int { return (int)(tile % CTd) * (PAIR ? 2 : 1) + (int)rank; };
    auto tile_mt = [&](long long tile) -> int { return (int)(tile / CTd); };
    long long t_lo, t_hi;
    const int kpart = p.kparts > 1 ? (int)(b % p.kparts) : 0;
    if (C::kStream && !p.whole_tiles) {
        t_lo = range_lo(n_tiles * U, G, b);
        t_hi = range_lo(n_tiles * U, G, b + 1);
    } else if (p.kparts > 1) {
        // the grid is exactly tiles x parts: one part of one tile per CTA (pair)
        const long long tile = b / p.kparts;
        t_lo = tile * U + (U * kpart) / p.kparts;
        t_hi = tile * U + (U * (kpart + 1)) / p.kparts;
    } else {
        t_lo = range_lo(n_tiles, G, b) * U;
        t_hi = range_lo(n_tiles, G, b + 1) * U;
    }

    // Every warpgroup takes part in the epilogue of the last tile (not with one row, which is one load per thread: the epilogue warps'
    // alone).  They meet the MMA warp at a named barrier of their own: a parity wait on d_full by the dequant warps, which may be
    // several short tiles ahead of the MMAs, could take an earlier tile's phase for the last one's.
    // Up to 6 rows of a tile that this CTA sums are the epilogue warps' alone if no partner's share is the partner's whole range (it
    // delivered early, or there is none): these warps then have everything before the last MMA, while the dequant warps would start
    // after it.  us, all warpgroups / epilogue warps: 1024 x 32768 int4 4 rows 13.7 / 12.6, 5 rows 14.4 / 13.3, 8 rows 14.4 / 13.4,
    // but 3072 x 12288 5 rows 12.7 / 13.5, 8 rows 12.7 / 13.7; with shares that are whole ranges 512 x 8192 8 rows 7.1 / 8.5.  (With
    // two passes in last_epilogue; by this rule and one pass 1024 x 32768 12.2, 12.9, 13.8, 3072 x 12288 12.7, 12.2, 512 x 8192 6.9.)
    bool spread_last = false;
    if (C::kStream && p.rows > 1 && t_lo < t_hi) {
        const long long first = div_nn(t_hi - 1, U) * U;               // the last tile's first unit
        spread_last = p.rows > 6 || t_lo > first || range_lo(n_tiles * U, G, b + 2) <= first + U;
    }
    constexpr uint32_t kSpreadThreads = (C::kWG + 1) * 128 + 32;
    static_assert(!C::kStream || C::kWG == 3, "last_epilogue: a warpgroup has at most NT / 16 groups of rows");

    if (warp == kWProducer || (C::kWProducers == 2 && warp == kWProducer2)) {
        // =========================== packed weights (+ scales / zeros): one thread per producer warp ===========================
        if (lane == 0) {
            // Without the promise that weight-side tensors are not written by the kernel before this one, nothing is read early.
            if (!p.overlap) ptx::grid_dependency_wait();
            // every box is copied whole (out-of-range parts are zero-filled)
            constexpr uint32_t kBytes = (uint32_t)WS::kBytes;
            const uint32_t mine = warp == kWProducer ? 0u : 1u;             // with two producers: the stages of this parity
            uint32_t si = 0, ws = 0, wph = 0;
            bool ok = true, ramped = false;
            for (long long t = t_lo; t < t_hi && ok;) {
                const long long tile = div_nn(t, U);                      // one 64-bit division per segment, none per unit
                const int u0 = (int)(t - tile * U);
                const int u1 = (int)min(U, u0 + (t_hi - t));
                const int ct = tile_ct(tile);
                for (int u = u0; u < u1; ++u, ++si) {
                    if (C::kWProducers == 1 || (si & 1u) == mine) {
                        // At the start all CTAs of the GPU ask for their whole rings at once, and the memory system serves
                        // the requests side by side: the first stage would arrive when a third of everything has (measured:
                        // 2.8 us after its copy was issued; 0.9 us for the luckiest CTA).  So the first stages go out alone,
                        // and the rest of the ring only once they have landed: each producer waits once, for the first
                        // stage it issued itself, before its second copy.
                        if (C::kStream && !ramped && si >= (uint32_t)C::kWProducers) {
                            if (!ptx::mbar_wait(ptx::smem_u32(&bars.w_full[mine]), 0u)) { atomicExch(p.status, 15); ok = false; break; }
                            ramped = true;
                        }
                        if (!ptx::mbar_wait(ptx::smem_u32(&bars.w_empty[ws]), wph ^ 1u)) { atomicExch(p.status, 11); ok = false; break; }
                        const uint32_t st = w_ring + ws * WS::kBytes, full = ptx::smem_u32(&bars.w_full[ws]);
                        ptx::mbar_arrive_expect_tx(full, kBytes);
                        ptx::tma_load_2d(st + WS::kW, &tm.w, ct * 128, u * H * F::WROWS, full);
                        if (SPARSE) ptx::tma_load_2d(st + WS::kMask, &tm.m, ct * 128, u * H * F::MROWS, full);
                        const int g0 = (int)p.gdiv((uint32_t)H * (uint32_t)u);
                        ptx::tma_load_2d(st + WS::kS, &tm.s, ct * 128, g0, full);
                        ptx::tma_load_2d(st + WS::kZ, &tm.z, ct * 128, g0, full);
                    }
                    if (++ws == C::kWStages) { ws = 0; wph ^= 1u; }
                }
                t += u1 - u0;
            }
        }
    } else if (PERM && warp == kBProducer) {
        // =========================== activation tiles in the permuted k order: the whole warp ===========================
        // The few valid rows are fetched with plain asynchronous 16-byte copies (eight consecutive k each) into a small
        // staging ring, kXStaging units ahead, every lane its own chunks.  When the unit's A / activation stage is free,
        // each lane reorders its chunks to (k0, k4, k1, k5, k2, k6, k3, k7), the order the dequant warps produce without
        // byte shuffles, and stores them at their place in the stage's 128-byte-swizzled tile; then the stage is
        // announced to the MMA warp.  Rows past the last valid one are zeroed once, up front.  (A tensor-map copy plus
        // a barrier per unit, as for the other formats, costs this warp more per unit than the unit may take.)
        for (uint32_t o = lane * 16; o < (uint32_t)(kABStages * kBStageBytes); o += 32 * 16) ptx::sts128(b_ring + o, make_uint4(0, 0, 0, 0));
        ptx::grid_dependency_wait();      // the activations may be the output of the kernel before this one in the stream
        if (lane == 0) ptx::grid_launch_dependents();      // as below
        constexpr int D = C::kXStaging;
        const int total = (int)(t_hi - t_lo);
        const int nrows = min(NT, p.rows);                              // (one row tile: these shapes have at most NT rows)
        const int n_chunks = nrows * 8 * H;                             // chunk index = row * (8 * H) + part * 8 + chunk of the part's 128-byte row segment
        int u_next = (int)(t_lo - div_nn(t_lo, U) * U);                // unit (within its column tile) of the next copy
        auto fetch = [&](int slot) {
            for (int idx = lane; idx < n_chunks; idx += 32) {
                const int r = idx / (8 * H), hc = idx % (8 * H);
                const int k = (u_next * H * 8 + hc) * 8;
                // past the end of the row (N is a multiple of 64, not of 256): zero fill
                ptx::cp_async_16(x_staging + slot * kBStageBytes + idx * 16, x + (size_t)r * p.N + (k < p.N ? k : 0), k < p.N ? 16u : 0u);
            }
            ptx::cp_async_commit();
            if (++u_next == (int)U) u_next = 0;
        };
        for (int j = 0; j < D - 1; ++j) {                                   // (always D - 1 groups, empty ones if need be: wait_group counts groups)
            if (j < total) fetch(j);
            else ptx::cp_async_commit();
        }
        for (int i = 0; i < total; ++i) {
            if (i + D - 1 < total) fetch((i + D - 1) % D);
            else ptx::cp_async_commit();                                  // (keeps the group count per iteration fixed)
            const uint32_t s = (uint32_t)(i % kABStages), ph = (uint32_t)(i / kABStages) & 1u;
            if (!ptx::mbar_wait(ptx::smem_u32(&bars.ab_free[s]), ph ^ 1u)) {
                if (lane == 0) atomicExch(p.status, 12);
                break;
            }
            ptx::cp_async_wait_group<D - 1>();                           // the copies of unit i (this lane's own chunks) have landed
            const uint32_t src = x_staging + (i % D) * kBStageBytes, dst = b_ring + s * kBStageBytes;
            for (int idx = lane; idx < n_chunks; idx += 32) {
                const int r = idx / (8 * H), hc = idx % (8 * H);
                const uint4 a = ptx::lds128(src + idx * 16);
                uint4 o;
                o.x = prmt(a.x, a.z, 0x5410);      // (k0, k4)
                o.y = prmt(a.x, a.z, 0x7632);      // (k1, k5)
                o.z = prmt(a.y, a.w, 0x5410);      // (k2, k6)
                o.w = prmt(a.y, a.w, 0x7632);      // (k3, k7)
                // 128-byte swizzle of the tile a tensor-map copy would have produced: chunk c of row r sits at c ^ (r % 8)
                ptx::sts128(dst + (hc >> 3) * kBHalfBytes + r * 128 + (((hc & 7) ^ (r & 7)) << 4), o);
            }
            ptx::fence_proxy_async_smem();         // the MMAs read the tile through the async proxy
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars.ab_full[s]));
        }
        ptx::cp_async_wait_group<0>();
    } else if (warp == kBProducer) {
        // =========================== activation tiles, one 64-k sub-tile per part of a unit: one thread ===========================
        if (lane == 0) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            // the activations may be the output of the kernel before this one in the stream (the weight-side tensors
            // are not: see the launch attribute in launch_nt)
            ptx::grid_dependency_wait();
            // The next kernel of the stream may be scheduled from here on (it takes an SM only when a CTA of this grid has
            // left it); if it is one of these kernels, its set-up and its first weight copies then overlap this grid's tail.
            // Not before the wait: see ptx.cuh.
            ptx::grid_launch_dependents();
            for (long long t = t_lo; t < t_hi && ok;) {
                const long long tile = div_nn(t, U);
                const int u0 = (int)(t - tile * U);
                const int u1 = (int)min(U, u0 + (t_hi - t));
                const int mt = tile_mt(tile);
                for (int u = u0; u < u1; ++u) {
                    if (!ptx::mbar_wait(ptx::smem_u32(&bars.ab_free[s]), ph ^ 1u)) { atomicExch(p.status, 12); ok = false; break; }
                    const uint32_t full = ptx::smem_u32(&bars.ab_full[s]);
                    if (PAIR) {
                        // both CTAs' halves are counted on the leader's barrier, which expects the bytes of both
                        const uint32_t lfull = ptx::map_to_cta(full, 0);
                        if (rank == 0) ptx::mbar_arrive_expect_tx(full, 2u * (uint32_t)kBStageBytes);
                        const int r0 = mt * NT + (int)rank * (NT / 2);
                        ptx::tma_load_2d_pair(b_ring + s * kBStageBytes, &tm.x, u * 128, r0, lfull);
                        ptx::tma_load_2d_pair(b_ring + s * kBStageBytes + kBHalfBytes, &tm.x, u * 128 + 64, r0, lfull);
                    } else if (C::kStream) {
                        // one copy per unit: H sub-tiles of 64 k, laid out one after the other
                        ptx::mbar_arrive_expect_tx(full, (uint32_t)kBStageBytes);
                        ptx::tma_load_3d(b_ring + s * kBStageBytes, &tm.x, 0, mt * NT, u * H, full);
                    } else {
                        ptx::mbar_arrive_expect_tx(full, (uint32_t)kBStageBytes);
                        ptx::tma_load_2d(b_ring + s * kBStageBytes, &tm.x, u * 128, mt * NT, full);
                        ptx::tma_load_2d(b_ring + s * kBStageBytes + kBHalfBytes, &tm.x, u * 128 + 64, mt * NT, full);
                    }
                    if (++s == kABStages) { s = 0; ph ^= 1u; }
                }
                t += u1 - u0;
            }
        }
    } else if (warp == kMma) {
        // =========================== MMA issuer: the warp walks the loop, one elected lane issues ===========================
        {
            const uint32_t idesc = PAIR ? ptx::idesc_f16_m256(NT) : ptx::idesc_f16_m128(NT);
            uint32_t si = 0, seg = 0;
            bool ok = true, last = false;
            if (PAIR && rank != 0) t_lo = t_hi;              // the leader issues for both CTAs
            for (long long t = t_lo; t < t_hi && ok;) {
                const long long tile = div_nn(t, U);
                const int u0 = (int)(t - tile * U);
                const int u1 = (int)min(U, u0 + (t_hi - t));
                last = t + (u1 - u0) >= t_hi;
                const uint32_t buf = seg % C::kDBufs, d = tmem_base + buf * C::kDCols;
                if (!ptx::mbar_wait(ptx::smem_u32(&bars.d_empty[buf]), ((seg / C::kDBufs) & 1u) ^ 1u)) {
                    if (lane == 0) atomicExch(p.status, 21);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                uint32_t s = si % kABStages, ph = (si / kABStages) & 1u;
                for (int u = u0; u < u1; ++u, ++si) {
                    if (!ptx::mbar_wait(ptx::smem_u32(&bars.ab_full[s]), ph)) {
                        if (lane == 0) atomicExch(p.status, 22);
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after_sync();
                    const uint64_t bdesc = ptx::smem_desc_sw128(b_ring + s * kBStageBytes);
                    const uint32_t a0 = tmem_base + C::kACol0 + s * C::kAStageCols;
                    if (ptx::elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4 * H; ++k) {
                            // K = 16 per instruction: +8 columns of A; B: +32 bytes (2 descriptor units) inside a 64-k sub-tile
                            const uint64_t bd = bdesc + (uint64_t)((k >> 2) * (kBHalfBytes >> 4) + (k & 3) * 2);
                            if (PAIR) ptx::umma_f16_ts_pair(d, a0 + k * 8, bd, idesc, (u > u0 || k > 0) ? 1u : 0u);
                            else ptx::umma_f16_ts(d, a0 + k * 8, bd, idesc, (u > u0 || k > 0) ? 1u : 0u);
                        }
                        if (PAIR) {                                      // the stage comes free in both CTAs
                            ptx::tc_commit_pair(ptx::map_to_cta(ptx::smem_u32(&bars.ab_free[s]), 0));
                            ptx::tc_commit_pair(ptx::map_to_cta(ptx::smem_u32(&bars.ab_free[s]), 1));
                        } else {
                            ptx::tc_commit(ptx::smem_u32(&bars.ab_free[s]));
                        }
                    }
                    __syncwarp();
                    if (++s == kABStages) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                if (ptx::elect_one()) {
                    if (PAIR) {
                        ptx::tc_commit_pair(ptx::map_to_cta(ptx::smem_u32(&bars.d_full), 0));
                        ptx::tc_commit_pair(ptx::map_to_cta(ptx::smem_u32(&bars.d_full), 1));
                    } else {
                        ptx::tc_commit(ptx::smem_u32(&bars.d_full));
                    }
                }
                __syncwarp();
                if (C::kStream) {
                    // the epilogue warps sleep on a hardware barrier instead of polling for the whole segment
                    if (!ptx::mbar_wait(ptx::smem_u32(&bars.d_full), seg & 1u)) {
                        if (lane == 0) atomicExch(p.status, 23);
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_before_sync();
                    if (spread_last && last) ptx::named_bar_arrive(5, kSpreadThreads);
                    else ptx::named_bar_arrive(2 + 4 * buf, 128 + 32);
                }
                ++seg;
                t += u1 - u0;
            }
            if (C::kStream && !ok) {
                s_abort = 1;
                __threadfence_block();
                if (!spread_last || !last) ptx::named_bar_arrive(2 + 4 * (seg % C::kDBufs), 128 + 32);
                if (spread_last) ptx::named_bar_arrive(5, kSpreadThreads);      // the last tile's: by every role once, whatever happened
            }
        }
    } else {
        // =========================== dequant warpgroups; epilogue warps ===========================
        // Accumulator of one finished tile (or K part of one) of the whole-tile shapes -> fp16 rows of `out`, or fp32 rows in the scratch.
        // (Weight streaming: early_epilogue, last_epilogue.)  Run by 4 warps whose index modulo 4 selects the 32 tensor-memory lanes
        // (= weight columns) they may read.
        bool dependency_waited = false;
        auto epilogue = [&](uint32_t seg, long long tile) -> bool {
            if (!dependency_waited) {
                // outputs, old outputs and the scratch may still be in use by the kernel before this one in the stream
                ptx::grid_dependency_wait();
                dependency_waited = true;
            }
            const int mt = tile_mt(tile), ct = tile_ct(tile);
            const int col = (warp & 3) * 32 + lane;
            const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
            const int scol = ct * 128 + col;
            const bool col_ok = scol < p.S;
            const int row0 = mt * NT;
            const int nrows = min(NT, p.rows - row0);
            // K parts: fp32 rows j0 .. of this lane's column into the (part, row, S) scratch; the reduce kernel sums the parts
            auto put_kpart = [&](auto& v, int j0) {
                constexpr int CNT = (int)(sizeof(v) / sizeof(uint32_t));
                if (!col_ok) return;
#pragma unroll
                for (int j = 0; j < CNT; ++j)
                    if (j0 + j < nrows)
                        p.partials[((size_t)kpart * p.rows + row0 + j0 + j) * p.S + scol] = __uint_as_float(v[j]);
            };
            bool got = ptx::mbar_wait(ptx::smem_u32(&bars.d_full), seg & 1u);
            if (!got && lane == 0) atomicExch(p.status, 33);
            // the four warps of an epilogue group meet at named barriers further down: a give-up has to be
            // the whole group's decision, or the warps that went on would wait there for ever
            if (!got) s_abort = 1;
            ptx::named_bar_sync(1 + 3 * ((warp - kEpiWarp0) >> 2), 128);
            got = s_abort == 0;
            if (!got) return false;
            ptx::tc_fence_after_sync();
            // matvec route with more than 64 rows (a batch of one-row products): the caller's old values of rows
            // j0 .. of this lane's column are added to the unrounded sums, so that there is still one rounding
            auto add_old_outs = [&](uint32_t (&v)[16], int j0) {
                if (!col_ok) return;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (j0 + j < nrows)
                        v[j] = __float_as_uint(__uint_as_float(v[j]) + __half2float(p.om.dst[0][(size_t)(row0 + j0 + j) * p.om.ld + p.om.col(scol)]));
            };
            // 16 accumulator columns (= 16 output rows) at a time: transposed through a 4 KB shared-memory tile so that
            // the global stores are 16-byte rows instead of one 2-byte element per lane
            const int eg = (warp - kEpiWarp0) >> 2;                     // epilogue warpgroup: its share of the accumulator columns
            const uint32_t stage_tile = epi_tile + eg * 4096;          // [16 rows][128 columns] fp16
            const uint32_t bar_id = 1 + 3 * eg;                         // named barriers 1 and 4
            const int t128 = (warp & 3) * 32 + lane;
            constexpr int kShare = NT / kEpiGroups;
            const int j_end = (eg + 1) * kShare;
            if (PAIR) {
                // A CTA of a pair has the shared memory to stage its whole share as fp16 ([kShare rows][128 columns]):
                // the accumulator is released after the tensor-memory loads and conversions alone, and the global
                // stores run while the next tile's MMAs are already under way.
                const uint32_t stage = epi_tile + eg * (kShare * 256);
#pragma unroll 1
                for (int j0 = eg * kShare; j0 < j_end; j0 += 16) {
                    uint32_t v[16];
                    ptx::tmem_ld16(lane_addr + j0, v);
                    ptx::tc_wait_ld();
                    if (j0 + 16 >= j_end) {
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&bars.d_empty[0]), 0));
                    }
                    if (p.kparts > 1) {
                        put_kpart(v, j0);
                        continue;
                    }
                    if (p.accumulate) add_old_outs(v, j0);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        ptx::sts16(stage + (j0 - eg * kShare + j) * 256 + col * 2,
                                   __half_as_ushort(__float2half_rn(__uint_as_float(v[j]))));
                }
                ptx::named_bar_sync(bar_id, 128);
#pragma unroll 1
                for (int idx = t128; idx < (p.kparts > 1 ? 0 : kShare * 16); idx += 128) {   // 16-byte chunks: row = idx / 16, chunk = idx % 16
                    const int m = eg * kShare + (idx >> 4), c8 = (idx & 15) * 8;
                    if (m < nrows && ct * 128 + c8 < p.S) {
                        const uint4 q = ptx::lds128(stage + (idx >> 4) * 256 + c8 * 2);
                        const size_t at = (size_t)(row0 + m) * p.om.ld + p.om.col(ct * 128 + c8);   // (a chunk of 8 columns never straddles parts)
                        for (int d = 0; d < p.om.n_dst; ++d) *reinterpret_cast<uint4*>(p.om.dst[d] + at) = q;
                    }
                }
                ptx::named_bar_sync(bar_id, 128);                       // the staging area may be written again
            } else
#pragma unroll 1
            for (int j0 = eg * kShare; j0 < j_end; j0 += 16) {
                uint32_t v[16];
                ptx::tmem_ld16(lane_addr + j0, v);
                ptx::tc_wait_ld();
                if (j0 + 16 >= j_end) {                // this group's last columns are in registers: its share of the accumulator is free
                    ptx::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars.d_empty[0]));
                }
                if (p.kparts > 1) {
                    put_kpart(v, j0);
                    continue;
                }
                if (p.accumulate) add_old_outs(v, j0);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    ptx::sts16(stage_tile + j * 256 + col * 2, __half_as_ushort(__float2half_rn(__uint_as_float(v[j]))));
                ptx::named_bar_sync(bar_id, 128);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int idx = t128 + r * 128;                     // 256 chunks of 16 bytes: row = idx / 16, chunk = idx % 16
                    const int m = j0 + (idx >> 4), c8 = (idx & 15) * 8;
                    if (m < nrows && ct * 128 + c8 < p.S) {
                        const uint4 q = ptx::lds128(stage_tile + (idx >> 4) * 256 + c8 * 2);
                        const size_t at = (size_t)(row0 + m) * p.om.ld + p.om.col(ct * 128 + c8);
                        for (int d = 0; d < p.om.n_dst; ++d) *reinterpret_cast<uint4*>(p.om.dst[d] + at) = q;
                    }
                }
                ptx::named_bar_sync(bar_id, 128);
            }
            // Stores into other GPUs' buffers: every storing thread makes its own stores visible system-wide before the
            // CTA can finish, so that the hand-shake kernel's flag (written by another SM, possibly over another link)
            // cannot reach a peer before this data has.
            if (p.om.n_dst > 1) __threadfence_system();
            return true;
        };

        // Weight-streaming shapes: where this CTA's last tile is and who shares it, by one warp while nothing has arrived yet.  (It is ~1500 cycles of
        // divisions.  Done by every warp before its last tile it cost up to 1 us where that tile is short: int4 16 rows 5120 x 5120 10.2 us, now 9.7,
        // 16:32 5120 x 20480 26.2 / 24.6, int4 48 rows 2048 x 8192 9.9 / 9.4, 128 rows 5120 x 20480 33.4 / 31.9.)
        if constexpr (C::kStream) {
            if (warp == kEpiWarp0 && t_lo < t_hi) {
                const long long tile = div_nn(t_hi - 1, U), lo_t = tile * U;
                TileCtas ctas{(int)b, (int)b, 1};
                if (t_lo > lo_t || t_hi < lo_t + U) {
                    ctas.b_lo = range_owner(n_tiles * U, G, lo_t);
                    ctas.b_hi = range_owner(n_tiles * U, G, lo_t + U - 1);
                    if (NT > 32) ctas.members = ctas.b_hi - ctas.b_lo + (range_lo(n_tiles * U, G, ctas.b_hi + 1) == lo_t + U ? 1 : 0);
                }
                if (lane == 0) s_last = {ctas, tile_ct(tile), tile_mt(tile), C::kDBufs == 1 ? 0u : (uint32_t)(tile - div_nn(t_lo, U)) % C::kDBufs};
            }
            ptx::named_bar_sync(7, (C::kWG + 1) * 128);
        }
        // One warp of every CTA that sums a shared tile with others; b_lo as it starts, the other members before their last tile
        auto settle_presence = [&](bool start) {
            if (warp != kEpiWarp0 || t_lo >= t_hi) return;
            const TileCtas ctas = s_last.ctas;
            if (ctas.members <= 1 || start != (b == ctas.b_lo)) return;
            ptx::grid_dependency_wait();                   // (the words may still be in use by the kernel before this one)
            if (start) {
#pragma unroll 1
                for (int r0 = 0; r0 < ctas.members; r0 += 32) {
                    const int r = r0 + lane;
                    const bool gone = r > 0 && r < ctas.members && atomicExch(p.present + b + r, 1u) == 2u;
                    if (gone) atomicExch(p.present + b + r, 0u);
                    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, gone);
                    if (lane == 0) s_left[r0 / 32] = bits;
                }
            } else if (lane == 0) {
                uint32_t seen;
                for (uint32_t spins = 0; (seen = atomicCAS(p.present + b, 0u, spins < kLeaveSpins ? 0u : 2u)) == 0u && spins < kLeaveSpins; ++spins) __nanosleep(500);
                if (seen != 0u) atomicExch(p.present + b, 0u);
                s_left[0] = seen == 0u;
            }
            __syncwarp();
        };

        uint32_t seg = 0;
        bool aborted = false;                                              // a wait timed out (weight-streaming shapes)
        if (warp >= kEpiWarp0 + 4 * kEpiGroups) {
            // (an epilogue warpgroup that this configuration does not use)
        } else if (warp >= kEpiWarp0) {
            // ----- dedicated epilogue warps: one pass per segment -----
            if constexpr (C::kStream && NT > 32) settle_presence(true);
            for (long long t = t_lo; t < t_hi;) {
                const long long tile = div_nn(t, U);
                const int u0 = (int)(t - tile * U);
                const int u1 = (int)min(U, u0 + (t_hi - t));
                if constexpr (C::kStream) {
                    if (t + (u1 - u0) >= t_hi) break;                  // the last tile: below
                    ptx::grid_dependency_wait();                       // as in `epilogue`
                    const int col = (int)threadIdx.x & 127, scol = tile_ct(tile) * 128 + col, row0 = tile_mt(tile) * NT, rows = min(NT, p.rows - row0);
                    const bool col_ok = scol < p.S;
                    const uint32_t buf = seg % C::kDBufs;
                    if (!early_epilogue<NT>(p.om, p.om.n_dst, p.om.ld, p.om.dst[0] + (size_t)row0 * p.om.ld + (col_ok ? p.om.col(scol) : 0), rows, col_ok ? rows : 0,
                                        p.accumulate, u0 == 0 ? nullptr : reinterpret_cast<uint4*>(p.partials) + (size_t)(C::kSlots * b) * C::kSlotVecs + col,
                                        tmem_base + buf * C::kDCols, 2 + 4 * buf, ptx::smem_u32(&bars.d_empty[buf]), ptx::smem_u32(const_cast<int*>(&s_abort)))) {
                        aborted = true;
                        break;
                    }
                } else if (!epilogue(seg, tile)) break;
                ++seg;
                t += u1 - u0;
            }
            if constexpr (C::kStream && NT > 32) {
                if (!aborted) settle_presence(false);
            }
        } else {
            // ----- dequant warps -----
            const int wg = warp >> 2;                                           // warpgroup: takes every kWG-th weight stage
            const int col = (warp & 3) * 32 + lane;                             // weight column in the tile = tensor-memory lane
            const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
            uint32_t si0 = 0;                                                    // si0: weight stages consumed before this segment
            // the stores into tensor memory are complete -> the stage may be read by the MMAs
            auto announce = [&](int stage) {
                ptx::tc_wait_st();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&bars.ab_full[stage]), 0));
                    else ptx::mbar_arrive(ptx::smem_u32(&bars.ab_full[stage]));
                }
            };
            bool ok = true;
            for (long long t = t_lo; t < t_hi && ok;) {
                const long long tile = div_nn(t, U);
                const int u0 = (int)(t - tile * U);
                const int u1 = (int)min(U, u0 + (t_hi - t));
                // a unit of this warpgroup: its place in the rings, and the wait for its weights
                struct Unit {
                    uint32_t si, ws, st, g0, as, aph;       // stage index, weight stage and its address, first group, A stage and its phase
                };
                auto next_unit = [&](int u, Unit& n) -> bool {
                    n.si = si0 + (uint32_t)(u - u0);
                    n.ws = n.si % C::kWStages;                                              // constants: multiply-shift, no division
                    const uint32_t wph = (n.si / C::kWStages) & 1u;
                    if (C::kWGuard && !ptx::mbar_wait(ptx::smem_u32(&bars.w_empty[n.ws]), wph ^ 1u)) {   // see Cfg::kWStages
                        if (lane == 0) atomicExch(p.status, 35);
                        return false;
                    }
                    if (!ptx::mbar_wait(ptx::smem_u32(&bars.w_full[n.ws]), wph)) {
                        if (lane == 0) atomicExch(p.status, 31);
                        return false;
                    }
                    n.st = w_ring + n.ws * WS::kBytes;
                    n.g0 = p.gdiv((uint32_t)H * (uint32_t)u);
                    n.as = n.si % kABStages;
                    n.aph = (n.si / kABStages) & 1u;
                    return true;
                };
                // row of part h's group in the stage's boxes of scales and zero-points
                auto group_row = [&](int u, uint32_t g0, int h) -> uint32_t {
                    return h == 0 ? 0u : p.gdiv((uint32_t)H * (uint32_t)u + (uint32_t)h) - g0;   // 0 .. H - 1
                };
                // after the last read of the weight stage
                auto release_weights = [&](uint32_t ws) {
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars.w_empty[ws]));
                };
                // before the first store into the A stage: it (and its activation tile) is free once the MMAs of its previous use have completed
                auto acquire_a_stage = [&](const Unit& n, bool free_early) -> bool {
                    if (!free_early && !ptx::mbar_wait(ptx::smem_u32(&bars.ab_free[n.as]), n.aph ^ 1u)) {
                        if (lane == 0) atomicExch(p.status, 32);
                        return false;
                    }
                    ptx::tc_fence_after_sync();
                    return true;
                };
                auto words = [&](const Unit& n, int h) -> uint32_t { return n.st + WS::kW + h * (F::WROWS * 512) + col * 4; };
                auto masks = [&](const Unit& n, int h) -> uint32_t { return n.st + WS::kMask + h * (F::MROWS * 512) + col * 4; };
                auto a_cols = [&](const Unit& n, int h) -> uint32_t { return lane_addr + C::kACol0 + n.as * C::kAStageCols + h * 32; };
                // Fast mode: scale signs clear, zero-points integers in [0, 512] (16:32: see kFastBound and kWideBound), for every column of the
                // warp in every group of the unit.
                constexpr uint32_t kBound = kFastBound<SPARSE>;
                // this warpgroup's units of the segment: those whose stage index is congruent to wg modulo kWG
                for (int u = u0 + (int)(((uint32_t)wg + (uint32_t)C::kWG - si0 % (uint32_t)C::kWG) % (uint32_t)C::kWG); u < u1; u += C::kWG) {
                    Unit n;
                    if (!next_unit(u, n)) { ok = false; break; }
                    if constexpr (C::kStream) {
                        uint32_t A[32];
                        // Few rows are bound by this loop: by its instructions (per unit ~700 a scheduler with the other roles', and the half-precision
                        // pipe alone is busy for 650 cycles) and by the waits between its steps.  So the mode is voted before anything is
                        // decoded, for two groups at a time, the parts are straight-line code without a branch in between, and a unit is
                        // announced as soon as it is written.  (With a branch per part on a new group, the vote at the last part, the other modes'
                        // 32 registers beside it, and the announcement put off to the warpgroup's next unit: one row 16384 x 16384 int4 37.2 us,
                        // 16:32 52.4, int3 40.5, int2 37.3; now 35.4, 51.0, 39.1, 33.0.  General mode, which decoded twice: 66, 111, 79, 71; now
                        // 52, 78, 60, 57.  Not better: the parts as a loop of two iterations (36.8, 52.9, 41.6, 36.4, with 35.9, 51.5, 39.1, 33.8 at the
                        // time); two warpgroups with 128 registers; an MMA warp, an accumulator and half-stages for each warpgroup.  The shapes below,
                        // which wait for other things, do not gain.)
                        uint32_t sp[H / 2], zp[H / 2], zi[H / 2], nf = 0;           // two parts' scales, zero-points, zero-points + 1024
#pragma unroll
                        for (int h = 0; h < H; h += 2) {
                            const uint32_t a0 = n.st + WS::kS + col * 2 + group_row(u, n.g0, h) * 256, a1 = n.st + WS::kS + col * 2 + group_row(u, n.g0, h + 1) * 256;
                            sp[h / 2] = prmt(ptx::lds_u16(a0), ptx::lds_u16(a1), 0x5410);
                            zp[h / 2] = prmt(ptx::lds_u16(a0 + H * 256), ptx::lds_u16(a1 + H * 256), 0x5410);
                        }
#pragma unroll
                        for (int i = 0; i < H / 2; ++i) {
                            zi[i] = hadd2_u(zp[i], kMagic1024);                    // (integer zero-points: their value in the low bits)
                            nf |= not_fast_bits<kBound>(sp[i], zp[i], zi[i]);
                        }
                        // A unit that is not in the fast mode, with a decision per part: rolled (one body of each mode in the instruction
                        // cache), half a part at a time, so that these modes do not set the register count of the straight-line code.  Its fast mode
                        // of 16:32 is the wide one.  (us, zero-points 128..255 by the general mode / by this one: 48 rows 16384 x 16384 85 / 71, 13824 x 5120
                        // 28.9 / 25.3, one row 16384 x 16384 80 / 68.)
                        // Every second group in the exponent coding, one row 16384 x 16384: by conversions int4 180, 16:32 192, int3 179, int2 126, now
                        // 70, 94, 76, 72.  (The other shapes keep the conversions: beside this mode their general one takes longer, int4 512 rows
                        // 5120 x 20480 106.6 / 109.6, int3 124.5 / 133.6.)
                        auto decode_by_part = [&]() {
#pragma unroll 1
                            for (int h = 0; h < H; ++h) {
                                const uint32_t at = n.st + WS::kS + col * 2 + group_row(u, n.g0, h) * 256;
                                const uint32_t s = ptx::lds_u16(at), z = ptx::lds_u16(at + H * 256), zi = hadd2_u(z, kMagic1024);
                                ColK c;
                                c.s2 = dup_lo(s);
                                c.z2 = dup_lo(z);
                                c.zb = SPARSE ? prmt(zi, zi, 0x0000) : 0u;
                                const bool fast = !__any_sync(0xFFFFFFFFu, (not_fast_bits<SPARSE ? kWideBound : kBound>(s, z, zi) & 0xFFFFu) != 0);
                                const bool lin = __all_sync(0xFFFFFFFFu, __hge(__ushort_as_half((unsigned short)s), __ushort_as_half(0)));
#pragma unroll 1
                                for (int half = 0; half < 2; ++half) {
                                    uint32_t A[16];
                                    if (fast) F::template decode<SPARSE ? MODE_WIDE : MODE_FAST>(words(n, h), masks(n, h), half, c, A, lut);
                                    else if (lin) F::template decode<MODE_GENERAL>(words(n, h), masks(n, h), half, c, A, lut);
                                    else F::template decode<MODE_EITHER>(words(n, h), masks(n, h), half, c, A, lut);
                                    ptx::tmem_st16(a_cols(n, h) + 16 * half, A);
                                }
                                if (h == H - 1) release_weights(n.ws);
                            }
                        };
                        if (__builtin_expect(__any_sync(0xFFFFFFFFu, nf != 0), 0)) {
                            if (!acquire_a_stage(n, false)) { ok = false; break; }
                            decode_by_part();
                        } else {
#pragma unroll
                            for (int h = 0; h < H; ++h) {
                                ColK c;
                                c.s2 = (h & 1) ? dup_hi(sp[h / 2]) : dup_lo(sp[h / 2]);
                                c.z2 = (h & 1) ? dup_hi(zp[h / 2]) : dup_lo(zp[h / 2]);
                                c.zb = SPARSE ? prmt(zi[h / 2], zi[h / 2], (h & 1) ? 0x2222 : 0x0000) : 0u;
                                decode_part<F, MODE_FAST>(words(n, h), masks(n, h), c, A, lut);
                                if (h == H - 1) release_weights(n.ws);
                                if (h == 0 && !acquire_a_stage(n, false)) { ok = false; break; }
                                ptx::tmem_st32(a_cols(n, h), A);
                            }
                        }
                    } else {
                        // polled before the first part is decoded, so that the answer costs no latency when it is needed
                        const bool free_early = ptx::mbar_test_wait(ptx::smem_u32(&bars.ab_free[n.as]), n.aph ^ 1u);
                        // scale and zero-point of this thread's column in row `row` of the stage's group box, both halves of a register
                        auto load_group = [&](uint32_t row, ColK& c) {
                            const uint32_t sz = ptx::lds32(n.st + WS::kS + row * 256 + (col & ~1) * 2) >> (16 * (col & 1));
                            const uint32_t zz = ptx::lds32(n.st + WS::kZ + row * 256 + (col & ~1) * 2) >> (16 * (col & 1));
                            c.s2 = prmt(sz, sz, 0x1010);
                            c.z2 = prmt(zz, zz, 0x1010);
                            c.zb = 0;
                        };
                        auto not_fast = [&](const ColK& c) -> uint32_t {
                            const uint32_t zr = hadd2_u(hadd2_u(c.z2, kMagic1024), H2_N1024), zlo = c.z2 & 0xFFFFu;
                            return ((zlo | ((zlo & 0x7FFFu) + kBound) | c.s2) & 0x8000u) | (zr ^ c.z2);
                        };
                        // (by a conversion and a multiply, 16:32 2048 rows 5120 x 20480 took 342.9 us, now 339.5)
                        auto zero_bytes = [&](ColK& c) {
                            if (SPARSE) {
                                const uint32_t zi = hadd2_u(c.z2, kMagic1024);         // (integer zero-points: their value in the low bits)
                                c.zb = prmt(zi, zi, 0x0000);
                            }
                        };
                        // The parts are decoded in the fast mode; whether every group of the unit really is in it is voted once, when the last group
                        // has been read and before the weight stage is released.  If not, the unit is decoded again with a decision per part (the
                        // stores are simply overwritten).
                        bool redo = false;
                        {
                            ColK c;
                            uint32_t cur_row = 0xFFFFFFFFu, nf = 0;
#pragma unroll
                            for (int h = 0; h < H; ++h) {
                                // scale and zero-point change only where the group does (warp-uniform)
                                const uint32_t row = group_row(u, n.g0, h);
                                if (row != cur_row) {
                                    cur_row = row;
                                    load_group(row, c);
                                    nf |= not_fast(c);
                                    zero_bytes(c);
                                }
                                if (h == H - 1 && __any_sync(0xFFFFFFFFu, nf != 0)) {
                                    redo = true;
                                    break;
                                }
                                uint32_t A[32];
                                decode_part<F, MODE_FAST>(words(n, h), masks(n, h), c, A, lut);
                                if (h == H - 1) release_weights(n.ws);
                                if (h == 0 && !acquire_a_stage(n, free_early)) { ok = false; break; }
                                ptx::tmem_st32(a_cols(n, h), A);
                            }
                        }
                        if (redo && ok) {
                            // (rolled loop: three decode bodies in the instruction cache, not three per part)
                            ptx::tc_wait_st();
                            ColK c;
                            uint32_t cur_row = 0xFFFFFFFFu;
#pragma unroll 1
                            for (int h = 0; h < H; ++h) {
                                const uint32_t row = group_row(u, n.g0, h);
                                if (row != cur_row) {
                                    cur_row = row;
                                    load_group(row, c);
                                }
                                uint32_t A[32];
                                if (!__any_sync(0xFFFFFFFFu, not_fast(c) != 0)) {
                                    zero_bytes(c);
                                    decode_part<F, MODE_FAST>(words(n, h), masks(n, h), c, A, lut);
                                } else {
                                    c.zb = 0;
                                    const bool lin = __hge(__ushort_as_half((unsigned short)(c.s2 & 0xFFFFu)), __ushort_as_half(0));
                                    if (__all_sync(0xFFFFFFFFu, lin)) decode_part<F, MODE_GENERAL>(words(n, h), masks(n, h), c, A, lut);
                                    else decode_part<F, MODE_SLOW>(words(n, h), masks(n, h), c, A, lut);
                                }
                                if (h == H - 1) release_weights(n.ws);
                                ptx::tmem_st32(a_cols(n, h), A);
                            }
                        }
                    }
                    if (!ok) break;
                    announce((int)n.as);
                }
                if (!ok) { aborted = true; break; }
                si0 += (uint32_t)(u1 - u0);
                t += u1 - u0;
            }
        }
        if constexpr (C::kStream) {
            if (aborted) {
                if (spread_last) ptx::named_bar_arrive(5, kSpreadThreads);
            } else if (spread_last || (warp >= kEpiWarp0 && t_lo < t_hi)) {
                // outputs, old outputs and the scratch may still be in use by the kernel before this one in the stream
                ptx::grid_dependency_wait();
                const TileCtas ctas = s_last.ctas;
                const uint32_t buf = C::kDBufs == 1 ? 0u : s_last.buf;
                const int col = (warp & 3) * 32 + lane, scol = s_last.ct * 128 + col, row0 = s_last.mt * NT;
                const bool col_ok = scol < p.S;
                auto run = [&](auto epilogue) {
                    epilogue(p.om, p.om.n_dst, p.om.ld, p.om.dst[0] + (size_t)row0 * p.om.ld + (col_ok ? p.om.col(scol) : 0), col_ok, min(NT, p.rows - row0),
                             p.accumulate, reinterpret_cast<uint4*>(p.partials) + col, p.status, ctas, p, s_left,
                             tmem_base + buf * C::kDCols + ((uint32_t)((warp & 3) * 32) << 16), spread_last ? warp >> 2 : 0, spread_last ? C::kWG + 1 : 1,
                             spread_last ? 5 : 2 + 4 * buf, spread_last ? kSpreadThreads : 128 + 32, ptx::smem_u32(const_cast<int*>(&s_abort)));
                };
                if constexpr (NT <= 32 && !PERM) run([](const auto&... a) { last_epilogue_call<NT>(a...); });
                else run([](const auto&... a) { last_epilogue<NT>(a...); });
            }
        }
    }

    // ---- teardown: every role ends up here, also after a timed-out wait ----
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    if (PAIR) ptx::cluster_sync_all();       // neither CTA's barriers or tensor memory may go while the other can still reach them
    if (warp == kMma) {
        if (PAIR) ptx::tmem_dealloc_pair(tmem_base, C::kTmemCols);
        else ptx::tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// Sums the K parts written by umma_kernel (fp32, (part, row, S)) in part order, rounds once to fp16, and puts the
// scratch back to all-zero (the split-K reduction of the few-row shapes relies on that).  8 columns per thread.
// (no __restrict__ here or on umma_kernel's activations: both kernels may start while the kernel that writes what they
// read is still running, and a restrict-qualified pointer would allow the compiler to load above griddepcontrol.wait)
__global__ void kparts_reduce_kernel(float* parts, const OutMap om, int rows, int S, int kparts) {
    // (launched with programmatic stream serialization: touches nothing before the kernel that wrote the parts has
    // completed, and lets the next kernel be scheduled from then on)
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int s8 = S / 8;
    const long long n8 = (long long)rows * s8;
    const size_t stride = (size_t)rows * S;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int f = 0; f < kparts; ++f) {
            float4* src = reinterpret_cast<float4*>(parts + f * stride + i * 8);
            const float4 a = src[0], c = src[1];
            acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
            acc[4] += c.x; acc[5] += c.y; acc[6] += c.z; acc[7] += c.w;
            src[0] = make_float4(0.f, 0.f, 0.f, 0.f);
            src[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __half2 h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __floats2half2_rn(acc[2 * j], acc[2 * j + 1]);
        const long long row = i / s8;
        const int c8 = (int)(i - row * s8) * 8;
        const size_t at = (size_t)row * om.ld + om.col(c8);
        for (int d = 0; d < om.n_dst; ++d) *reinterpret_cast<uint4*>(om.dst[d] + at) = *reinterpret_cast<uint4*>(h);
    }
    if (om.n_dst > 1) __threadfence_system();        // as in umma_kernel's epilogue
}

// ---- host side -------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, found at run time so that the library does not link against libcuda.
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess && ptr)
            fn = (EncodeTiledFn)ptr;
        if (!fn) {
            (void)cudaGetLastError();
            void* h = dlopen("libcuda.so.1", RTLD_NOW | RTLD_GLOBAL);
            if (h) fn = (EncodeTiledFn)dlsym(h, "cuTensorMapEncodeTiled");
        }
    }
    return fn;
}

// The encoder needs a context that is current in the calling thread, which the first CUDA call of a new thread may find missing.
template <class Encode>
bool encode_with_context(Encode encode) {
    if (encode() == CUDA_SUCCESS) return true;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return encode() == CUDA_SUCCESS;
}

// 2-D row-major tensor (rows, cols) of `elem_bytes` elements, box (box_rows, box_cols)
bool encode_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t rows, uint64_t cols,
               uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swz) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * elem_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode_with_context([&] {
        return enc(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    });
}

// what the last tcgen05 launch of this host thread chose: tile rows + 1000 if CTA pairs + 10000 * K parts (tests read it)
thread_local int g_last_shape = 0;
thread_local int g_last_schedule = 0;             // i4mm_last_launch_schedule

// Encoded tensor maps are a pure function of (base address, shape, box, swizzle): callers multiply with the same
// weight tensors over and over, so the maps are kept in a small direct-mapped table instead of being encoded by the
// driver five times per call (which costs more host time than the launch itself).
struct MapKey {
    const void* base;
    uint64_t rows, cols;
    uint32_t box_rows, box_cols;
    int dt, elem_bytes, swz;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && box_rows == o.box_rows && box_cols == o.box_cols &&
               dt == o.dt && elem_bytes == o.elem_bytes && swz == o.swz;
    }
};
struct MapSlot {
    MapKey key;
    CUtensorMap map;
    bool valid;
};
constexpr int kMapSlots = 512;
std::mutex g_map_mutex;
MapSlot g_map_cache[kMapSlots];

bool encode_2d_cached(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t rows, uint64_t cols,
                      uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swz) {
    const MapKey key{base, rows, cols, box_rows, box_cols, (int)dt, elem_bytes, (int)swz};
    uint64_t h = (uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull;
    h ^= (rows * 0xC2B2AE3D27D4EB4Full) ^ (cols << 17) ^ ((uint64_t)box_rows << 40) ^ ((uint64_t)box_cols << 52) ^ (uint64_t)dt;
    MapSlot& slot = g_map_cache[(h >> 32) % kMapSlots];
    {
        std::lock_guard<std::mutex> lock(g_map_mutex);
        if (slot.valid && slot.key == key) {
            *out = slot.map;
            return true;
        }
    }
    if (!encode_2d(out, base, dt, elem_bytes, rows, cols, box_rows, box_cols, swz)) return false;
    std::lock_guard<std::mutex> lock(g_map_mutex);
    slot.key = key;
    slot.map = *out;
    slot.valid = true;
    return true;
}

// The activations (rows, N) of the weight-streaming shapes seen as (N / 64 blocks, rows, 64 k): one copy fetches the
// `blocks` consecutive 64-k sub-tiles of a unit, each box_rows x 128 bytes in the 128-byte swizzle, one after the other.
bool encode_x_blocks_cached(CUtensorMap* out, const void* base, uint64_t rows, uint64_t n, uint32_t box_rows, uint32_t blocks) {
    const MapKey key{base, rows, n, box_rows, blocks, -3, 2, (int)CU_TENSOR_MAP_SWIZZLE_128B};
    uint64_t h = (uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull;
    h ^= (rows * 0xC2B2AE3D27D4EB4Full) ^ (n << 17) ^ ((uint64_t)box_rows << 40) ^ ((uint64_t)blocks << 52) ^ 0x33ull;
    MapSlot& slot = g_map_cache[(h >> 32) % kMapSlots];
    {
        std::lock_guard<std::mutex> lock(g_map_mutex);
        if (slot.valid && slot.key == key) {
            *out = slot.map;
            return true;
        }
    }
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(n / 64)};
    const cuuint64_t strides[2] = {(cuuint64_t)n * 2, 128};
    const cuuint32_t box[3] = {64, box_rows, blocks};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (!encode_with_context([&] {
            return enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        }))
        return false;
    std::lock_guard<std::mutex> lock(g_map_mutex);
    slot.key = key;
    slot.map = *out;
    slot.valid = true;
    return true;
}

// Shapes of whole tiles (more than 64 rows), where these fill less than half of the GPU: cut K into parts so that
// tiles x parts CTAs (pairs) run, as long as every part keeps at least 4 stages and the partial outputs fit the scratch.
int choose_kparts(long long capacity, long long tiles, int U, long long rows, long long S) {
    if (tiles <= 0 || tiles * 2 > capacity) return 1;
    long long f = capacity / tiles;
    if (f > 8) f = 8;
    if (f > U / 4) f = U / 4;
    while (f > 1 && f * rows * S * 4 > (long long)kPartialBytes) --f;
    return f < 2 ? 1 : (int)f;
}

int launch_kparts_reduce(const UmmaParams& p, cudaStream_t stream, cudaError_t* cuda_err) {
    const long long n8 = (long long)p.rows * p.S / 8;
    long long blocks = (n8 + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)blocks, 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kparts_reduce_kernel, p.partials, p.om, p.rows, p.S, p.kparts);
    if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
    count_launch();
    return I4MM_OK;
}

// Weight-streaming shapes: whole tiles, although some SMs then have less to do or nothing, where the units that the busiest CTA has more than
// with equal ranges cost less than the sums of shared tiles (units: 256 k, from 65 rows on 128 k; us, int4, equal ranges / whole tiles):
// 16 rows 2048 x 15360 (1.5 units more) 10.9 / 9.6, 5120 x 15360 (3.8) 16.4 / 16.1, 2048 x 7680 (4.8) 8.7 / 8.5, 5120 x 14080 (5.1) 15.5 / 16.1,
// 2048 x 25600, two tiles a CTA (5.2) 13.9 / 14.8; 64 rows 5120 x 14080 18.3 / 18.0, 8192 x 15360 (6.1) 24.6 / 24.7, 2048 x 25600 17.8 / 16.6;
// 128 rows 2048 x 9600 (7.9) 14.0 / 12.9, 5120 x 14080 (10.3) 22.8 / 22.1, 5120 x 12800 (13.0) 21.4 / 22.0, 2048 x 25600 (10.4) 25.1 / 22.9;
// 72 rows 5120 x 14080 21.0 / 21.2.
bool whole_tiles_better(int nt, long long tiles, int U, long long ctas) {
    if (tiles % ctas == 0) return false;                       // (equal ranges are whole tiles)
    const long long w = (tiles + ctas - 1) / ctas;
    const long long tenths = 10 * (w * U * ctas - tiles * U) / ctas;
    return tenths < (nt <= 32 ? 45 : nt <= 64 ? (w == 1 ? 55 : 75) : (w == 1 ? 105 : 140));
}

// Weight-streaming shapes: how many CTAs share each tile, the same number for all, or 0: all CTAs have equal ranges and tiles are shared as it
// comes.  Equal ranges use every SM, but a CTA of them may hold parts of two tiles, one summed after the other, and few tiles have many
// partners, each of which costs its share of the sums: a smaller grid in which no range crosses a tile is the faster one wherever the
// units that it adds cost less.  Costs in tenths of a unit's time, fitted to 1366 shapes (int4, int3, 16:32; 1 .. 128 rows; 4 .. 64 tiles of
// 1024 .. 20480 rows of weights), where the rule takes 0.92 (up to 16 rows), 0.89, 0.90 and 0.86 (65 rows and more) of the time of equal
// ranges in the mean; none is slower by more than 4 %, three by more than 1.2 %.
// us, equal ranges / CTAs per tile: int4, 4 rows 3072 x 1024 7.0 / 6.0 (6), 2048 x 2560 6.7 / 6.0 (3), 16 rows 4096 x 1024 8.9 / 6.8 (8), 32 rows
// 2048 x 2560 8.7 / 7.3 (3), 64 rows 4096 x 1024 11.1 / 8.2 (8), 128 rows 4096 x 8192 17.2 / 14.5 (2), 4096 x 5120 13.7 / 12.5 (3), 2048 x 1024
// 11.5 / 8.3 (4); not taken: 4 rows 13824 x 2560 11.6 / 11.8 (6), 5120 x 2560 (3) 8.7 / 8.9, 20480 x 5120 19.8 / 21.3 (3).
int ctas_of_a_tile(int nt, bool sparse, long long tiles, long long U, long long ctas) {
    const long long partner = nt <= 16 ? (sparse ? 2 : 4) : nt <= 32 ? (sparse ? 4 : 5) : nt <= 64 ? (sparse ? 4 : 6) : 6;
    const long long two_tiles = nt <= 32 ? 10 : nt <= 64 ? 12 : 44;
    if (tiles * 2 > ctas) return 0;
    const long long most = ctas / tiles < U ? ctas / tiles : U;
    long long least = tiles * U < ctas ? 10 : 10 * tiles * U / ctas;
    const long long shared_by = 10 * ctas / tiles < 10 * U ? 10 * ctas / tiles : 10 * U;
    least += partner * shared_by / 10 + two_tiles;
    int best = 0;
    for (long long k = 2; k <= most; ++k) {
        const long long cost = 10 * ((U + k - 1) / k) + partner * k;
        if (cost < least) { least = cost; best = (int)k; }
    }
    return best;
}

template <int BITS, bool SPARSE, int NT, bool PAIR, bool PERM = false, bool STREAM = NT <= 64>
int launch_nt(const UmmaParams& p_in, const __half* x, int n_groups, cudaStream_t stream, cudaError_t* cuda_err) {
    UmmaParams p = p_in;
    p.kparts = 1;
    using F = UFormat<BITS, SPARSE>;
    using C = Cfg<NT, PAIR, STREAM>;
    constexpr int H = C::kHalves;
    p.U = (p.N + 64 * H - 1) / (64 * H);
    constexpr int kBStageBytes = H * (PAIR ? NT / 2 : NT) * 128;
    TensorMaps tm;
    const uint64_t R = SPARSE ? (uint64_t)p.N / 16 : (uint64_t)p.N * BITS / 32;
    bool ok = C::kStream ? encode_x_blocks_cached(&tm.x, x, p.rows, p.N, NT, H)
                         : encode_2d_cached(&tm.x, x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.rows, p.N, PAIR ? NT / 2 : NT, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    ok = ok && encode_2d_cached(&tm.w, p.matrix, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, R, p.S, H * F::WROWS, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (SPARSE)
        ok = ok && encode_2d_cached(&tm.m, p.mask, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, (uint64_t)p.N / 32, p.S, H * F::MROWS, 128,
                             CU_TENSOR_MAP_SWIZZLE_NONE);
    else
        tm.m = tm.w;
    ok = ok && encode_2d_cached(&tm.s, p.scales, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, n_groups, p.S, H, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    ok = ok && encode_2d_cached(&tm.z, p.zeros, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, n_groups, p.S, H, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (!ok) return I4MM_ERR_DEVICE;

    const size_t smem = 1024 + (size_t)ABStages<NT, PAIR, STREAM>::value * kBStageBytes + (size_t)C::kWStages * WStage<F, H>::kBytes +
                        (C::kStream ? 0 : PAIR ? NT * 256 : 4096 * ((C::kEpiGroups == 2 && NT < 256) ? 2 : 1)) +
                        (PERM ? (size_t)C::kXStaging * kBStageBytes : 0);
    auto kern = umma_kernel<BITS, SPARSE, NT, PAIR, PERM, STREAM>;
    // per-device cache; atomic because two host threads may make their first call at once (both then compute the same value)
    static std::atomic<int> sm_count[16];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
    dev &= 15;
    if (sm_count[dev] == 0) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
        sm_count[dev] = sms;
    }
    if (PAIR) {
        // clusters of two CTAs; as many as can be resident at once, each walking its share of the pair tiles
        static std::atomic<int> max_clusters[16];
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.blockDim = dim3(C::kThreads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        if (max_clusters[dev] == 0) {
            cfg.gridDim = dim3(2 * (sm_count[dev] / 2), 1, 1);
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
                (void)cudaGetLastError();
                n = sm_count[dev] / 2;
            }
            if (n > sm_count[dev] / 2) n = sm_count[dev] / 2;
            max_clusters[dev] = n;
        }
        long long clusters = max_clusters[dev];
        const long long tiles2 = (long long)p.MTILES * ((p.CT + 1) / 2);
        if (!p.accumulate && !p.whole_tiles)
            p.kparts = choose_kparts(clusters, tiles2, p.U, p.rows, p.S);
        const long long work = tiles2 * p.kparts;
        if (clusters > work || p.kparts > 1) clusters = work;
        cfg.gridDim = dim3((unsigned)(2 * clusters), 1, 1);
        e = cudaLaunchKernelEx(&cfg, kern, tm, p, x);
        if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
        count_launch();
        g_last_shape = NT + 1000 + 10000 * (p.kparts > 1 ? p.kparts : 0);
        g_last_schedule = p.kparts > 1 ? I4MM_SCHEDULE_K_PARTS : I4MM_SCHEDULE_WHOLE_TILES;
        if (p.kparts > 1) return launch_kparts_reduce(p, stream, cuda_err);
        return I4MM_OK;
    }
    const long long n_tiles = (long long)p.MTILES * p.CT;
    long long grid = sm_count[dev];                     // one CTA per SM: every configuration fills its shared or tensor memory
    int schedule = I4MM_SCHEDULE_STREAM_EQUAL_RANGES;
    if (!C::kStream && !p.accumulate && !p.whole_tiles)
        p.kparts = choose_kparts(grid, n_tiles, p.U, p.rows, p.S);
    if (C::kStream) {
        p.whole_tiles = whole_tiles_better(NT, n_tiles, p.U, grid);
        if (p.whole_tiles) {
            const long long w = (n_tiles + grid - 1) / grid;
            grid = (n_tiles + w - 1) / w;
            schedule = I4MM_SCHEDULE_STREAM_WHOLE_TILES;
        } else if (const int k = ctas_of_a_tile(NT, SPARSE, n_tiles, p.U, grid)) {
            grid = n_tiles * k;
            schedule = I4MM_SCHEDULE_STREAM_CTAS_PER_TILE + k;
        }
    }
    const long long work = p.kparts > 1 ? n_tiles * p.kparts : C::kStream && !p.whole_tiles ? n_tiles * p.U : n_tiles;
    if (grid > work || p.kparts > 1) grid = work;
    constexpr long long kMostCtas = kPartialBytes / (C::kSlots * C::kSlotVecs * 16);       // those whose shares the scratch holds
    static_assert(!C::kStream || kMostCtas >= 148, "every SM of the GPU has its slots");
    static_assert(NT <= 32 || !C::kStream || (kMostCtas <= 32 * kLeftWords && kMostCtas * 4 <= kStatusOffset), "last_epilogue: a bit and a word per CTA");
    if (C::kStream && grid > kMostCtas) grid = kMostCtas;
    {
        // The kernel may start while the kernel before it in the stream is still running: its set-up overlaps that
        // kernel's tail, and with `overlap` so do its copies of the weight-side tensors (which the caller has declared
        // not to be written by that kernel).  Everything else waits for that kernel inside (griddepcontrol.wait).
        // Without the attribute a pass cost ~2 us more (one row: int4 5120 x 5120 16.4 -> 14.4 us with its zero-fill,
        // 16384 x 16384 44.3 -> 42.5; 48 rows of 13824 x 5120 28.7 -> 26.6).
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3((unsigned)grid, 1, 1);
        cfg.blockDim = dim3(C::kThreads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, tm, p, x);
    }
    if (e != cudaSuccess) { *cuda_err = e; return I4MM_ERR_LAUNCH; }
    count_launch();
    g_last_shape = NT + 10000 * (p.kparts > 1 ? p.kparts : 0);
    g_last_schedule = p.kparts > 1 ? I4MM_SCHEDULE_K_PARTS : C::kStream ? schedule : I4MM_SCHEDULE_WHOLE_TILES;
    if (p.kparts > 1) return launch_kparts_reduce(p, stream, cuda_err);
    return I4MM_OK;
}

// Rows per tile (the MMA's N).  Few rows: the smallest tile that holds them.  Many rows: the tile height that
// minimises (waves of tiles over the SMs) x (time per tile), so that e.g. 320 tiles of 256 rows (2.2 waves on 148
// SMs) become 440 tiles of 192 rows (3.0 waves) when that is faster.
int choose_tile_rows(int rows, int col_tiles, int sms, int max_nt) {
    if (rows <= 16) return 16;
    if (rows <= 32) return 32;
    if (rows <= 64) return 64;
    if (rows <= 128) return 128;
    const int cand[4] = {256, 224, 192, 160};
    int best = max_nt < 256 ? 192 : 256;
    long long best_cost = -1;
    for (int i = 0; i < 4; ++i) {
        const int nt = cand[i];
        if (nt > max_nt) continue;
        const long long tiles = (long long)((rows + nt - 1) / nt) * col_tiles;
        const long long waves = (tiles + sms - 1) / sms;
        const long long cost = waves * (nt + 24);          // + per-tile fill / drain, in row units
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = nt; }
    }
    return best;
}

constexpr int kPairMinRows = 128;

// More than 128 rows in one call: tiles of 128 rows on the weight-streaming shape, or taller ones on CTA pairs.  Pairs decode a weight for up
// to 256 rows at once and run a tile's MMAs on two SMs, so they win wherever their tiles fill the pairs; the streaming shape hands out single
// units, so it wins where they do not, and where pairs would cut K into parts that a second kernel adds up.  Both times in 1/100 us (units: 128 k;
// pairs: a fixed part, a quarter of a row per unit and row of the tile, the adding kernel; streaming: whole tiles, or equal ranges and their
// sums), fitted to 472 shapes of 130..512 rows (2048 / 5120 / 13824 x 2048..20480) and held against 160 more, drawn from 129..2048 rows and
// 1024..20480 on both sides: there the chosen one took 0.88 (int4), 0.87 (int3), 0.78 (int2) and 0.91 (16:32) of the time of pairs alone in the
// mean, within 1 % of always taking the better one, and was in no shape more than 1.5 % slower than pairs.
// us, pairs / streaming, int4: 13824 x 2048 200 rows 31.2 / 19.5 (K parts), 13824 x 5120 200 rows 48.6 / 34.7, 5120 x 5120 160 rows 24.6 / 18.9;
// 5120 x 6976 333 rows 27.0 / 32.9 (56 pair tiles of 192 rows leave 18 of 74 pairs idle, and are the faster ones all the same: the streaming shape
// decodes every weight three times).  (Where launch_nt then takes the same number of CTAs for every tile, it does so because that is faster than
// the equal ranges reckoned with here.)
bool streaming_better(bool sparse, int rows, int CT, int U, long long S, int sms, bool kparts_allowed) {
    const long long pairs = sms / 2, CT2 = (CT + 1) / 2, tiles = (long long)((rows + 127) / 128) * CT;
    const long long nt = choose_tile_rows(rows, (int)CT2, (int)pairs, 256), tiles2 = (rows + nt - 1) / nt * CT2;
    const long long kp = kparts_allowed ? choose_kparts(pairs, tiles2, U, rows, S) : 1;
    const long long t_pairs = 800 + (tiles2 * kp + pairs - 1) / pairs * ((U + kp - 1) / kp) * nt / 4 + (kp > 1 ? 1100 : 0);
    const long long w = (tiles + sms - 1) / sms;
    const long long t_streaming = tiles % sms == 0 || whole_tiles_better(128, tiles, U, sms) ? 800 + (sparse ? 45 : 40) * w * U + 300 * (w - 1)
                                                                                             : 1000 + (sparse ? 55 : 46) * tiles * U / sms;
    return t_streaming * 20 < t_pairs * 19;
}

template <int BITS, bool SPARSE>
int launch_fmt(UmmaParams& p, const __half* x, int n_groups, int pair_mode, int force_nt, cudaStream_t stream, cudaError_t* cuda_err) {
    static std::atomic<int> sms_of[16];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    dev &= 15;
    int sms = sms_of[dev].load();
    if (sms == 0) {
        int n = 0;
        sms = (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) ? n : 148;
        sms_of[dev].store(sms);
    }
    // 128 rows or more (the whole-tile configurations) run as CTA pairs, two SMs per MMA, unless the caller asked for single CTAs
    const bool pair = pair_mode == 0 && (force_nt ? force_nt >= 128 : p.rows >= kPairMinRows);
    // 65..128 rows: the weight-streaming shape, or whole tiles of the shape that is made for them (its decode does not share the CTA with sums,
    // and its stores are 16 bytes) where those leave fewer SMs idle than the sums cost.  us, whole tiles / streaming: int4 96 rows 2048 x 16384
    // 13.2 / 13.7, 16:32 14.7 / 16.0, 5120 x 16384 22.3 / 22.4, 26.0 / 28.0; K parts, as before / streaming: 5120 x 5120 21.4 / 13.8, 22.2 / 14.8,
    // 13824 x 5120 31.4 / 22.2, 34.7 / 23.6; two waves / streaming: 5120 x 20480 40.3 / 31.4, 47.4 / 37.0.
    // 128 rows in a CTA pair take 0.85 of the time per unit: pairs / streaming, int4, 5120 x 27648 (68 units to 58, of 128 k) 39.1 / 42.0, 13824 x 15360
    // (92 to 88) 53.6 / 56.7, 2048 x 20480 (27 to 17) 21.3 / 22.4, 5120 x 11008 (34 to 23) 22.2 / 20.3, 5120 x 20480 (68 to 43) 39.3 / 33.7.
    // With the same number of CTAs for every tile: 2048 x 5120 (14 to 6, 3 CTAs a tile) 11.9 / 10.5, 2048 x 6976 (14 to 8, 2 CTAs) 12.1 / 12.3.
    if (!force_nt && p.rows > 64 && p.rows <= 128 && p.om.n_dst == 1) {
        const long long U = (p.N + 127) / 128, w = (p.CT + sms - 1) / sms;
        const int k = pair ? ctas_of_a_tile(128, SPARSE, p.CT, U, sms) : 0;
        p.whole_tiles = p.CT % sms == 0 || (k ? w * U * 17 < ((U + k - 1) / k + 5 + k / 2) * 20
                                            : pair ? w * U * 17 * sms < (p.CT * U + 10 * sms) * 20 : whole_tiles_better(128, p.CT, (int)U, sms));
        if (!p.whole_tiles) {
            p.MTILES = 1;
            return launch_nt<BITS, SPARSE, 128, false, false, true>(p, x, n_groups, stream, cuda_err);
        }
    }
    if (!force_nt && pair_mode == 0 && p.rows > 128 && p.om.n_dst == 1 && streaming_better(SPARSE, p.rows, p.CT, (p.N + 127) / 128, p.S, sms, !p.accumulate)) {
        p.MTILES = (p.rows + 127) / 128;
        return launch_nt<BITS, SPARSE, 128, false, false, true>(p, x, n_groups, stream, cuda_err);
    }
    // Stores into several GPUs' buffers (the gathering multiply) make the epilogue of a tile last longer than the tile's
    // MMAs.  Under exactly that condition the CTA-pair instances with 224 and 256 rows per tile (two dequant warpgroups,
    // three weight stages) were seen, on 8 GPUs, to produce now and then one wrong block of 32 columns x one row tile
    // (one warp's weights of one 128-k unit); the 192-row pair instance (four warpgroups, six stages) and the single-CTA
    // 224 / 256 instances were not, and no run with one destination ever was.  The cause has not been found, so the
    // gathering multiply keeps to tiles of at most 192 rows when it runs as CTA pairs.
    const int max_nt = (pair && p.om.n_dst > 1) ? 192 : 256;
    const int nt = force_nt ? force_nt : pair ? choose_tile_rows(p.rows, (p.CT + 1) / 2, sms / 2, max_nt) : choose_tile_rows(p.rows, p.CT, sms, 256);
    p.MTILES = (p.rows + nt - 1) / nt;
    if (pair) {
        switch (nt) {
            case 128: return launch_nt<BITS, SPARSE, 128, true>(p, x, n_groups, stream, cuda_err);
            case 160: return launch_nt<BITS, SPARSE, 160, true>(p, x, n_groups, stream, cuda_err);
            case 192: return launch_nt<BITS, SPARSE, 192, true>(p, x, n_groups, stream, cuda_err);
            case 224: return launch_nt<BITS, SPARSE, 224, true>(p, x, n_groups, stream, cuda_err);
            case 256: return launch_nt<BITS, SPARSE, 256, true>(p, x, n_groups, stream, cuda_err);
            default: break;
        }
    }
    switch (nt) {
        case 16:
            // Up to 3 rows of dense int4: the k order that needs no byte shuffles.  More rows cost the one warp that reorders the
            // activations more per unit than the unit takes, the sooner the more units a CTA has (us, this order / the natural one:
            // 16384 x 16384 1 row 37.4 / 39.5, 3 rows 39.1 / 40.0, 4 rows 41.9 / 40.0, 5 rows 45.0 / 40.3; 13824 x 5120 3 rows 15.6 / 16.5,
            // 4 rows 16.0 / 16.4, 5 rows 16.8 / 16.9; 5120 x 20480 3 rows 19.8 / 20.6, 4 rows 20.6 / 20.4; 1024 x 32768 5 rows 12.3 / 12.9;
            // the other way round only where a tile is one or two units: 512 x 8192 3 rows 6.7 / 6.5)
            if (BITS == 4 && !SPARSE && p.rows <= 3) return launch_nt<BITS, SPARSE, 16, false, BITS == 4 && !SPARSE>(p, x, n_groups, stream, cuda_err);
            return launch_nt<BITS, SPARSE, 16, false>(p, x, n_groups, stream, cuda_err);
        case 32: return launch_nt<BITS, SPARSE, 32, false>(p, x, n_groups, stream, cuda_err);
        case 64: return launch_nt<BITS, SPARSE, 64, false>(p, x, n_groups, stream, cuda_err);
        case 128: return launch_nt<BITS, SPARSE, 128, false>(p, x, n_groups, stream, cuda_err);
        case 160: return launch_nt<BITS, SPARSE, 160, false>(p, x, n_groups, stream, cuda_err);
        case 192: return launch_nt<BITS, SPARSE, 192, false>(p, x, n_groups, stream, cuda_err);
        case 224: return launch_nt<BITS, SPARSE, 224, false>(p, x, n_groups, stream, cuda_err);
        default: return launch_nt<BITS, SPARSE, 256, false>(p, x, n_groups, stream, cuda_err);
    }
}

}  // namespace

int umma_last_shape() { return g_last_shape; }
int umma_last_schedule() { return g_last_schedule; }
void set_last_shape(int shape) {
    g_last_shape = shape;
    g_last_schedule = 0;
}

bool umma_supported(int bits, bool sparse, int total_rows, int N, int S) {
    (void)bits; (void)sparse; (void)S;
    return total_rows >= 1 && N >= 64 && encode_tiled_fn() != nullptr;
}

int umma_launch(int bits, bool sparse, const StreamParams& sp, int total_rows, int n_groups, int group_size, int cta_pairs /* 0 by shape, 1 never */,
                int force_nt /* 0 = by shape */, int overlap, cudaStream_t stream, cudaError_t* cuda_err) {
    (void)group_size;
    UmmaParams p{};
    p.om = sp.om;
    p.matrix = sp.matrix;
    p.mask = sp.mask;
    p.scales = sp.scales;
    p.zeros = sp.zeros;
    p.partials = sp.partials;
    p.present = sp.counters;
    p.status = sp.status;
    p.rows = total_rows;
    p.N = sp.N;
    p.S = sp.S;
    p.U = 0;                      // set per configuration (units of 128 k or 256 k)
    p.CT = sp.CT;
    p.accumulate = sp.accumulate;
    p.overlap = overlap;
    p.gdiv = sp.gdiv;
    if (sparse) return launch_fmt<4, true>(p, sp.x, n_groups, cta_pairs, force_nt, stream, cuda_err);
    if (bits == 4) return launch_fmt<4, false>(p, sp.x, n_groups, cta_pairs, force_nt, stream, cuda_err);
    if (bits == 3) return launch_fmt<3, false>(p, sp.x, n_groups, cta_pairs, force_nt, stream, cuda_err);
    return launch_fmt<2, false>(p, sp.x, n_groups, cta_pairs, force_nt, stream, cuda_err);
}

}  // namespace i4mm
