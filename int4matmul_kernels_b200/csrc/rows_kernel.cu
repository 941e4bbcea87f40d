// A few activation rows (up to 8) times a small matrix on the warp-level tensor instruction.
//
// Replaces MVA_Int4_Half (matvec_kernel.cu:198-267) for one row and MMA_Int4_Half (matmul_kernel.cu:219-333) for 2..8,
// where a launch of the tcgen05 kernel is mostly its fixed cost (barrier and tensor-memory set-up, one producer thread
// filling the rings, hand-over between warps, the split-K tail).  A warp owns 64 weight columns and walks K in steps of
// 128: lane 4 g + t holds the 32-block of k number t of the step for the columns 4 g .. 4 g + 3 (and 32 further on),
// which is what 16-byte pieces of the packed rows are, and it is also a legal A operand of mma.sync m16n8k16 (16 weight
// columns x 16 k; which k a lane's registers stand for is free as long as the activation operand agrees).  So the packed
// words go from global memory through the lane's own 16 bytes of a shared-memory ring (asynchronous copies, no block
// barrier), are decoded in registers and feed the tensor instruction directly: no weight tile, no producer warp.
//
// A CTA is 4 warps over the same 64 columns, each taking every 4th step; their sums meet in shared memory.  Where there
// are fewer 64-column tiles than CTAs fit on the GPU (4 per SM), K is cut into parts, one CTA each, whose sums meet in
// scratch in a fixed order (results are bit-reproducible).
//
// What bounds it: per packed dense int4 word 5 ALU and 8 half-precision instructions, all of which issue every second
// cycle on this GPU (measured stand-alone: 19.8 cycles a word and scheduler with the mma; here ~30), and the copies: 16-byte
// asynchronous copies without any arithmetic stream 3.7 TB/s, which is why large matrices stay with the tcgen05 kernel
// and its tensor-map copies (rule and figures at rows_supported).
#include "../../include/int4matmul_b200.h"

#include <atomic>

#include "common.cuh"
#include "dequant.cuh"
#include "ptx.cuh"

namespace i4mm {

namespace {

constexpr int kKLanes = 4;                           // warps of a CTA: all over the same columns, every 4th step each
constexpr int kSets = 2;                             // 32-column sets of a warp
constexpr int kCtasPerSm = 4;                        // (4 warps x 4 CTAs: 2 x 8 and 8 x 2 were 1..20 % slower, 24 warps of 80 registers too)
constexpr int kTileCols = 32 * kSets;                // S is a multiple of 64, so column tiles are never ragged
constexpr int kRowsThreads = 32 * kKLanes;
constexpr int kMaxRows = 8;                          // the N dimension of m16n8k16

struct RowsParams {
    OutMap om;
    const uint32_t* matrix;
    const uint32_t* mask;
    const __half* x;
    const __half* scales;
    const __half* zeros;
    unsigned long long* partials;    // one partial tile per CTA: [row][64 columns] of (fp32 value | tag 1 << 32)
    int* status;
    int rows, N, S;
    int U;                           // 128-k steps per tile
    int tiles;                       // column tiles
    int parts;                       // CTAs that share a tile's K
    int accumulate, overlap;
    GroupDiv gdiv;
};

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// (plain shared-memory reads: the compiler may schedule them freely between the barriers)
__device__ __forceinline__ uint4 s128(const unsigned char* p) { return *reinterpret_cast<const uint4*>(p); }

__device__ __forceinline__ void cp_async_16_zfill(uint32_t dst, const void* src, bool valid) {
    ptx::cp_async_16(dst, src, valid ? 16u : 0u);
}

// ---- formats: a lane's 32-block of one column, in chunks ---------------------------------------------------------
// kLoads    16-byte loads (4 columns each) of packed rows per 32-block; kMaskLoads of mask rows
// kChunks   pieces a 32-block is decoded in; kPairs fp16 pairs per column and piece
// load      the packed words a chunk needs; decode: one column's pairs; first / second: which k of the chunk's
//           2 * kPairs ones pair p stands for (low and high half)
template <int BITS, bool SPARSE>
struct RFormat;

template <>
struct RFormat<4, false> {
    static constexpr int kLoads = 4, kMaskLoads = 0, kChunks = 4, kPairs = 4;
    struct Words { uint4 w; };
    __device__ static __forceinline__ void load(const unsigned char* st, int chunk, Words& o) { o.w = s128(st + chunk * 512); }
    // nibbles j and j + 4 sit at the same offset of the word's two 16-bit halves: one LOP3 plants both
    __host__ __device__ static constexpr int first(int p) { return p; }
    __host__ __device__ static constexpr int second(int p) { return p + 4; }
    template <int MODE>
    __device__ static __forceinline__ void decode(Words& o, int, const uint32_t*, int col, const ColK& c, uint32_t (&A)[kPairs]) {
        const uint32_t w = (&o.w.x)[col], w8 = w >> 8;
        const uint32_t off1 = hsub2_u(BASE_1_1, c.z2), off16 = hsub2_u(H2_N64, c.z2);
        A[0] = finish<4, MODE>(and_or(w, 0x000F000Fu, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
        A[1] = finish<4, MODE>(and_or(w, 0x00F000F0u, kMagic1024), H2_1_16, H2_N64, off16, c);
        A[2] = finish<4, MODE>(and_or(w8, 0x000F000Fu, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
        A[3] = finish<4, MODE>(and_or(w8, 0x00F000F0u, kMagic1024), H2_1_16, H2_N64, off16, c);
    }
};

template <>
struct RFormat<2, false> {
    static constexpr int kLoads = 2, kMaskLoads = 0, kChunks = 2, kPairs = 8;
    struct Words { uint4 w; };
    __device__ static __forceinline__ void load(const unsigned char* st, int chunk, Words& o) { o.w = s128(st + chunk * 512); }
    __host__ __device__ static constexpr int first(int p) { return p; }
    __host__ __device__ static constexpr int second(int p) { return p + 8; }
    template <int MODE>
    __device__ static __forceinline__ void decode(Words& o, int, const uint32_t*, int col, const ColK& c, uint32_t (&A)[kPairs]) {
        const uint32_t w = (&o.w.x)[col], w8 = w >> 8;
        const uint32_t off1 = hsub2_u(BASE_1_1, c.z2), off4 = hsub2_u(H2_N256, c.z2), off16 = hsub2_u(H2_N64, c.z2),
                       off64 = hsub2_u(H2_N16, c.z2);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t v = h ? w8 : w;
            A[4 * h + 0] = finish<2, MODE>(and_or(v, 0x00030003u, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
            A[4 * h + 1] = finish<2, MODE>(and_or(v, 0x000C000Cu, kMagic1024), H2_1_4, H2_N256, off4, c);
            A[4 * h + 2] = finish<2, MODE>(and_or(v, 0x00300030u, kMagic1024), H2_1_16, H2_N64, off16, c);
            A[4 * h + 3] = finish<2, MODE>(and_or(v, 0x00C000C0u, kMagic1024), H2_1_64, H2_N16, off64, c);
        }
    }
};

template <>
struct RFormat<3, false> {
    static constexpr int kLoads = 3, kMaskLoads = 0, kChunks = 1, kPairs = 16;
    struct Words { uint4 w0, w1, w2; };
    __device__ static __forceinline__ void load(const unsigned char* st, int, Words& o) {
        o.w0 = s128(st);
        o.w1 = s128(st + 512);
        o.w2 = s128(st + 1024);
    }
    // ten fields of the 96-bit stream at a time: fields i and i + 5 brought to the same offset of two 16-bit halves
    __host__ __device__ static constexpr int first(int p) { return p < 15 ? p / 5 * 10 + p % 5 : 30; }
    __host__ __device__ static constexpr int second(int p) { return p < 15 ? p / 5 * 10 + p % 5 + 5 : 31; }
    template <int MODE>
    __device__ static __forceinline__ void decode(Words& o, int, const uint32_t*, int col, const ColK& c, uint32_t (&A)[kPairs]) {
        const uint32_t w0 = (&o.w0.x)[col], w1 = (&o.w1.x)[col], w2 = (&o.w2.x)[col];
        const uint32_t off1 = hsub2_u(BASE_1_1, c.z2), off8 = hsub2_u(H2_N128, c.z2), off64 = hsub2_u(H2_N16, c.z2);
        const uint32_t ten[3] = {w0, __funnelshift_r(w0, w1, 30), __funnelshift_r(w1, w2, 28)};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t y = bit_select(0x00007FFFu, ten[i], ten[i] << 1), y9 = y >> 9;
            A[5 * i + 0] = finish<3, MODE>(and_or(y, 0x00070007u, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
            A[5 * i + 1] = finish<3, MODE>(and_or(y, 0x00380038u, kMagic1024), H2_1_8, H2_N128, off8, c);
            A[5 * i + 2] = finish<3, MODE>(and_or(y, 0x01C001C0u, kMagic1024), H2_1_64, H2_N16, off64, c);
            A[5 * i + 3] = finish<3, MODE>(and_or(y9, 0x00070007u, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
            A[5 * i + 4] = finish<3, MODE>(and_or(y9, 0x00380038u, kMagic1024), H2_1_8, H2_N128, off8, c);
        }
        const uint32_t u = w2 >> 26;
        A[15] = finish<3, MODE>(and_or(bit_select(0x00000007u, u, u << 13), 0x00070007u, kMagic1024), MUL_1_1, BASE_1_1, off1, c);
    }
};

template <>
struct RFormat<4, true> {
    static constexpr int kLoads = 2, kMaskLoads = 1, kChunks = 4, kPairs = 4;
    struct Words { uint4 lo, hi, m; };
    __host__ __device__ static constexpr int first(int p) { return 2 * p; }
    __host__ __device__ static constexpr int second(int p) { return 2 * p + 1; }
    __device__ static __forceinline__ void load(const unsigned char* st, int chunk, Words& o) {
        if (chunk == 0) {
            o.lo = s128(st);
            o.hi = s128(st + 512);
            o.m = s128(st + 1024);
        }
    }
    template <int MODE>
    __device__ static __forceinline__ void decode(Words& o, int chunk, const uint32_t* lut, int col, const ColK& c, uint32_t (&A)[kPairs]) {
        sparse_expand<MODE>((&o.lo.x)[col], (&o.hi.x)[col], (&o.m.x)[col], chunk, lut, c, A);
    }
};

// One stage of a warp's ring: per 32-column set the packed words [load][lane] x 16 B; the scales and zeros of the step's
// two 64-k halves (64 columns each); the activations [row][16 chunks of 8 k] (chunks permuted so that the 8 x 4 lanes'
// reads of 16 bytes hit different banks).
template <class F, int R>
struct RStage {
    static constexpr int kSet = (F::kLoads + F::kMaskLoads) * 512;
    static constexpr int kScale = kSets * kSet;                        // [half][64 columns] fp16
    static constexpr int kZero = kScale + 128 * kSets;
    static constexpr int kX = kZero + 128 * kSets;
    static constexpr int kBytes = kX + R * 256;
};
__device__ __forceinline__ uint32_t x_chunk(uint32_t row, uint32_t c) { return c ^ (c >> 3) ^ ((row & 1u) << 1); }

// Shared memory of a CTA (kCtasPerSm share an SM's 228 KB, of which each costs 1 KB by itself): the K lanes' sums (with 5..8
// rows half of the lanes at a time) and the rings.
template <class F, int R>
struct RSmem {
    static constexpr int kRedLanes = R > 4 ? kKLanes / 2 : kKLanes;
    static constexpr int kRed = kRedLanes * R * kTileCols * 4;
    static constexpr int kFit = ((228 / kCtasPerSm - 1) * 1024 - (F::kMaskLoads ? 1024 : 0) - kRed) / kKLanes / RStage<F, R>::kBytes;
    static constexpr int kDepth = kFit > 4 ? 4 : kFit;
    static constexpr int kBytes = kRed + kKLanes * kDepth * RStage<F, R>::kBytes;
};

// The lane's 32 k of one activation row, paired like the format's weights.  x_row: the row's 16 chunks of the stage
template <class F>
__device__ __forceinline__ void load_x(const unsigned char* x_row, uint32_t row, uint32_t t, uint32_t (&B)[16]) {
    uint32_t X[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 q = s128(x_row + x_chunk(row, t * 4 + i) * 16);
        X[4 * i] = q.x; X[4 * i + 1] = q.y; X[4 * i + 2] = q.z; X[4 * i + 3] = q.w;
    }
    constexpr int P = F::kPairs;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int a = i / P * (2 * P) + F::first(i % P), c = i / P * (2 * P) + F::second(i % P);
        B[i] = (a + 1 == c && a % 2 == 0) ? X[a / 2]
                                          : prmt(X[a / 2], X[c / 2], ((a & 1) ? 0x32u : 0x10u) | ((c & 1) ? 0x7600u : 0x5400u));
    }
}

// One set (32 columns) x 128 k.  words: this lane's packed words of the set
template <class F, int MODE>
__device__ __forceinline__ void compute_set(const unsigned char* words, const uint32_t* lut, const ColK (&ck)[4], const uint32_t (&B)[16],
                                            float (&c)[2][4]) {
    typename F::Words w;
#pragma unroll
    for (int ch = 0; ch < F::kChunks; ++ch) {
        F::load(words, ch, w);
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) {
            uint32_t A0[F::kPairs], A1[F::kPairs];
            F::template decode<MODE>(w, ch, lut, 2 * cp, ck[2 * cp], A0);
            F::template decode<MODE>(w, ch, lut, 2 * cp + 1, ck[2 * cp + 1], A1);
#pragma unroll
            for (int i = 0; i < F::kPairs; i += 2)
                mma_16816(c[cp], A0[i], A1[i], A0[i + 1], A1[i + 1], B[ch * F::kPairs + i], B[ch * F::kPairs + i + 1]);
        }
    }
}

__device__ __forceinline__ void column_constants(uint2 s4, uint2 z4, ColK (&ck)[4]) {
    ck[0].s2 = dup_lo(s4.x); ck[1].s2 = dup_hi(s4.x); ck[2].s2 = dup_lo(s4.y); ck[3].s2 = dup_hi(s4.y);
    ck[0].z2 = dup_lo(z4.x); ck[1].z2 = dup_hi(z4.x); ck[2].z2 = dup_lo(z4.y); ck[3].z2 = dup_hi(z4.y);
#pragma unroll
    for (int i = 0; i < 4; ++i) ck[i].zb = 0;
}

// Two columns x 128 k outside the fast mode: columns 2 cp and 2 cp + 1 of the lane's four (cp may be a run-time value).
template <class F, int MODE>
__device__ __forceinline__ void compute_pair(const unsigned char* words, const uint32_t* lut, int cp, uint32_t s, uint32_t z,
                                             const uint32_t (&B)[16], float (&c)[4]) {
    ColK ck[2];
    ck[0].s2 = dup_lo(s); ck[1].s2 = dup_hi(s);
    ck[0].z2 = dup_lo(z); ck[1].z2 = dup_hi(z);
    ck[0].zb = ck[1].zb = 0;
    typename F::Words w;
#pragma unroll
    for (int ch = 0; ch < F::kChunks; ++ch) {
        F::load(words, ch, w);
        if (ch == 0 || F::kMaskLoads == 0) {                 // (the sparse format loads once and consumes its words)
            uint4* const q = reinterpret_cast<uint4*>(&w);
#pragma unroll
            for (int i = 0; i < (int)(sizeof(w) / sizeof(uint4)); ++i) {
                q[i].x = cp ? q[i].z : q[i].x;
                q[i].y = cp ? q[i].w : q[i].y;
            }
        }
        uint32_t A0[F::kPairs], A1[F::kPairs];
        F::template decode<MODE>(w, ch, lut, 0, ck[0], A0);
        F::template decode<MODE>(w, ch, lut, 1, ck[1], A1);
#pragma unroll
        for (int i = 0; i < F::kPairs; i += 2) mma_16816(c, A0[i], A1[i], A0[i + 1], A1[i + 1], B[ch * F::kPairs + i], B[ch * F::kPairs + i + 1]);
    }
}

// R: rows the shared memory is laid out for (the launch's rows are at most R)
template <int BITS, bool SPARSE, int R>
__global__ void __launch_bounds__(kRowsThreads, kCtasPerSm) rows_kernel(const RowsParams p) {
    using F = RFormat<BITS, SPARSE>;
    using ST = RStage<F, R>;
    using SM = RSmem<F, R>;
    constexpr int D = SM::kDepth;
    static_assert(D >= 2, "a ring needs two stages");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t lut_mem[SPARSE ? 256 : 1];
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
    const int g = lane >> 2, t = lane & 3, kl = warp;
    float* const red = reinterpret_cast<float*>(smem_raw);                          // [K lane][row][64]
    unsigned char* const ring = smem_raw + SM::kRed + warp * (D * ST::kBytes);
    const uint32_t ring_addr = ptx::smem_u32(ring);

    // Without the promise that weight-side tensors are not written by the kernel before this one, nothing is read early
    if (!p.overlap) ptx::grid_dependency_wait();

    // ---- this CTA's steps: one part of one tile's K, or (more tiles than CTAs) several whole tiles.  Consecutive CTAs take
    // consecutive tiles, so that the CTAs of a part walk down the same packed rows together ----
    const int part = p.parts > 1 ? (int)blockIdx.x / p.tiles : 0;
    int t_lo, n_steps;
    if (p.parts > 1) {
        const int base = ((int)blockIdx.x - part * p.tiles) * p.U;
        t_lo = base + (int)((long long)p.U * part / p.parts);
        n_steps = base + (int)((long long)p.U * (part + 1) / p.parts) - t_lo;
    } else {
        const int lo = (int)range_lo(p.tiles, gridDim.x, blockIdx.x);
        t_lo = lo * p.U;
        n_steps = ((int)range_lo(p.tiles, gridDim.x, blockIdx.x + 1) - lo) * p.U;
    }
    const int first_tile = t_lo / p.U;

    // ---- copies: position of the next step to fetch, for this warp ----
    const size_t row_bytes = (size_t)p.S * 4;
    const int n_blk = p.N >> 5, n_half = p.N >> 6;
    int f_pos = kl;                                    // index within the CTA's range
    int f_tile = first_tile, f_u = t_lo - first_tile * p.U + kl;
    const char *w_src, *m_src = nullptr;               // this lane's first packed / mask word of the step
    auto locate = [&]() {
        while (f_u >= p.U) { f_u -= p.U; ++f_tile; }
        const size_t col = (size_t)(f_tile * kTileCols + 4 * g) * 4;
        w_src = reinterpret_cast<const char*>(p.matrix) + (size_t)((4 * f_u + t) * F::kLoads) * row_bytes + col;
        if (SPARSE) m_src = reinterpret_cast<const char*>(p.mask) + (size_t)(4 * f_u + t) * row_bytes + col;
    };
    locate();
    auto fetch_weights = [&](int stage) {
        if (f_pos >= n_steps) return;
        const uint32_t st = ring_addr + stage * ST::kBytes;
        // a step that is only half there (N % 128 = 64) is zero-filled, scales and zero-points too
        const bool there = 4 * f_u + t < n_blk;
        const char* src = there ? w_src : reinterpret_cast<const char*>(p.matrix);
        const uint32_t n = there ? 16u : 0u;
#pragma unroll
        for (int j = 0; j < F::kLoads; ++j) {
#pragma unroll
            for (int set = 0; set < kSets; ++set) ptx::cp_async_16(st + set * ST::kSet + j * 512 + lane * 16, src + set * 128, n);
            if (j + 1 < F::kLoads) src += there ? row_bytes : 0;
        }
        if (SPARSE) {
            const char* msrc = there ? m_src : reinterpret_cast<const char*>(p.mask);
#pragma unroll
            for (int set = 0; set < kSets; ++set) ptx::cp_async_16(st + set * ST::kSet + F::kLoads * 512 + lane * 16, msrc + set * 128, n);
        }
        if (lane < 16 * kSets) {
            // lanes 0..15 the scales, 16..31 the zero-points: two 64-k halves x 8 chunks of 8 columns
            constexpr int kChunks = 4 * kSets;
            const int half = 2 * f_u + ((lane / kChunks) & 1);
            const bool ok = half < n_half;
            const __half* src_h = (lane < 2 * kChunks ? p.scales : p.zeros) + (size_t)p.gdiv((uint32_t)(ok ? half : 0)) * p.S + f_tile * kTileCols + (lane % kChunks) * 8;
            cp_async_16_zfill(st + ST::kScale + lane * 16, src_h, ok);
        }
    };
    auto fetch_x = [&](int stage) {
        if (f_pos >= n_steps) return;
        const uint32_t st = ring_addr + stage * ST::kBytes + ST::kX;
#pragma unroll
        for (int i0 = 0; i0 < R * 16; i0 += 32) {
            const int i = i0 + lane, row = i >> 4, c = i & 15;
            if (row < p.rows) {
                const int k = f_u * 128 + c * 8;
                cp_async_16_zfill(st + row * 256 + x_chunk(row, c) * 16, p.x + (size_t)row * p.N + (k < p.N ? k : 0), k < p.N);
            }
        }
    };
    auto fetch_advance = [&]() {
        f_pos += kKLanes;
        f_u += kKLanes;
        if (f_u >= p.U) {
            locate();
        } else {
            w_src += (size_t)(4 * kKLanes * F::kLoads) * row_bytes;
            if (SPARSE) m_src += (size_t)(4 * kKLanes) * row_bytes;
        }
    };

    // ---- prologue: all D stages ----
    if (p.overlap) {
        // the weight side of the first stages goes out before the kernel before this one has finished
        const int s_pos = f_pos, s_u = f_u, s_tile = f_tile;
#pragma unroll 1
        for (int j = 0; j < D; ++j) { fetch_weights(j); fetch_advance(); }
        f_pos = s_pos; f_u = s_u; f_tile = s_tile;
        locate();
        ptx::grid_dependency_wait();
#pragma unroll 1
        for (int j = 0; j < D; ++j) { fetch_x(j); fetch_advance(); ptx::cp_async_commit(); }
    } else {
#pragma unroll 1
        for (int j = 0; j < D; ++j) { fetch_weights(j); fetch_x(j); fetch_advance(); ptx::cp_async_commit(); }
    }
    ptx::grid_launch_dependents();                           // not before the wait: see ptx.cuh
    if (SPARSE) {
        for (int i = threadIdx.x; i < 256; i += kRowsThreads) lut_mem[i] = sparse_selectors(i);
        __syncthreads();
    }

    float acc[kSets][2][4];                            // set x column pair (4 g, 4 g + 1), (4 g + 2, 4 g + 3) x rows 2 t, 2 t + 1
#pragma unroll
    for (int i = 0; i < kSets * 8; ++i) (&acc[0][0][0])[i] = 0.f;

    const uint32_t xrow = (uint32_t)min(g, p.rows - 1);   // rows past the last one only feed accumulator columns nobody reads
    // ---- the K lanes' sums of one tile, and the tile's other CTAs' ----
    bool ok = true;
    auto flush = [&](int tile) {
        float* const mine = red + ((kl % SM::kRedLanes) * R) * kTileCols + 4 * g;
        __syncthreads();                                     // the previous tile's sums have been read
#pragma unroll
        for (int ph = kKLanes / SM::kRedLanes - 1; ph >= 0; --ph) {
            if (kl / SM::kRedLanes == ph) {
#pragma unroll
                for (int i = 0; i < kSets * 8; ++i) {
                    const int set = i >> 3, cp = (i >> 2) & 1, row = 2 * t + (i & 1);
                    float* const at = mine + row * kTileCols + set * 32 + 2 * cp + ((i >> 1) & 1);
                    if (row < p.rows) *at = acc[set][cp][i & 3] + (ph != kKLanes / SM::kRedLanes - 1 ? *at : 0.f);
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < kSets * 8; ++i) acc[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
        for (int i = threadIdx.x; i < p.rows * kTileCols; i += kRowsThreads) {
            const int row = i / kTileCols, c = i % kTileCols;
            const float* r0 = red + row * kTileCols + c;
            float v = r0[0];
#pragma unroll
            for (int j = 1; j < SM::kRedLanes; ++j) v += r0[j * R * kTileCols];
            if (part != p.parts - 1) {
                // an element of a partial tile is one 64-bit word (value | tag), written with one store; the reader clears it
                ptx::st_relaxed_gpu_u64(p.partials + ((size_t)blockIdx.x * kMaxRows + row) * kTileCols + c, (1ull << 32) | __float_as_uint(v));
                continue;
            }
            // the last part's CTA adds the others' sums in part order (their blocks have lower numbers, so they were started before it)
            for (int q = 0; q < p.parts - 1; q += 4) {
                unsigned long long w[4];
                unsigned long long* const src = p.partials + ((size_t)(q * p.tiles + tile) * kMaxRows + row) * kTileCols + c;
                const size_t step = (size_t)p.tiles * kMaxRows * kTileCols;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (q + j < p.parts - 1) w[j] = ptx::ld_relaxed_gpu_u64(src + j * step);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (q + j >= p.parts - 1) break;
                    for (uint32_t spins = 0; (uint32_t)(w[j] >> 32) != 1u && ok; ++spins) {
                        if (spins >= ptx::kSpinLimit) {            // a contributor never delivered: report, stop waiting
                            atomicExch(p.status, 36);
                            ok = false;
                            break;
                        }
                        __nanosleep(32);
                        w[j] = ptx::ld_relaxed_gpu_u64(src + j * step);
                    }
                    v += __uint_as_float((uint32_t)w[j]);
                    ptx::st_relaxed_gpu_u64(src + j * step, 0ull);
                }
            }
            const size_t at = (size_t)row * p.om.ld + p.om.col(tile * kTileCols + c);
            if (p.accumulate) v += __half2float(p.om.dst[0][at]);
            const __half h = __float2half_rn(v);
            for (int d = 0; d < p.om.n_dst; ++d) p.om.dst[d][at] = h;
        }
    };

    int pos = kl, stage = 0, tile = first_tile;
    for (int seg_lo = 0; seg_lo < n_steps; ++tile) {
        const int seg_end = min((tile + 1) * p.U - t_lo, n_steps);
        for (; pos < seg_end; pos += kKLanes) {
            ptx::cp_async_wait_group<D - 1>();            // this step's copies have landed (own chunks), ...
            __syncwarp();                                    // ... and the other lanes' (scales, zeros, activations)
            const unsigned char* const st = ring + stage * ST::kBytes;
            const unsigned char* const x_row = st + ST::kX + xrow * 256;
            const unsigned char* const s_row = st + ST::kScale + (t >> 1) * (64 * kSets) + g * 8;
            const unsigned char* const z_row = st + ST::kZero + (t >> 1) * (64 * kSets) + g * 8;
            uint2 s4[kSets], z4[kSets];
            uint32_t nf = 0;
#pragma unroll
            for (int set = 0; set < kSets; ++set) {
                s4[set] = *reinterpret_cast<const uint2*>(s_row + set * 64);
                z4[set] = *reinterpret_cast<const uint2*>(z_row + set * 64);
                // fast mode: scale signs clear, zero-points integers in [0, 512] ([0, 127] for the sparse format)
                constexpr uint32_t kAdd = SPARSE ? 0x280F280Fu : 0x1FFF1FFFu;
                auto not_fast = [&](uint32_t s, uint32_t z) {
                    return ((z | s | ((z & 0x7FFF7FFFu) + kAdd)) & 0x80008000u) | (hadd2_u(hadd2_u(z, kMagic1024), H2_N1024) ^ z);
                };
                nf |= not_fast(s4[set].x, z4[set].x) | not_fast(s4[set].y, z4[set].y);
            }
            uint32_t B[16];
            load_x<F>(x_row, xrow, t, B);
            if (!__any_sync(0xFFFFFFFFu, nf != 0)) {
#pragma unroll
                for (int set = 0; set < kSets; ++set) {
                    ColK ck[4];
                    column_constants(s4[set], z4[set], ck);
                    if (SPARSE) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) ck[i].zb = __half2uint_rz(__ushort_as_half((unsigned short)(ck[i].z2 & 0xFFFFu))) * 0x01010101u;
                    }
                    compute_set<F, MODE_FAST>(st + set * ST::kSet + lane * 16, lut_mem, ck, B, acc[set]);
                }
            } else {
                // (rolled, so that these modes do not set the register count of the main loop)
#pragma unroll 1
                for (int i = 0; i < 2 * kSets; ++i) {
                    const int set = i >> 1, cp = i & 1;
                    const uint32_t s = *reinterpret_cast<const uint32_t*>(s_row + set * 64 + cp * 4), z = *reinterpret_cast<const uint32_t*>(z_row + set * 64 + cp * 4);
                    const unsigned char* const words = st + set * ST::kSet + lane * 16;
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
                    if (__all_sync(0xFFFFFFFFu, (s & 0x80008000u) == 0)) compute_pair<F, MODE_GENERAL>(words, lut_mem, cp, s, z, B, c);
                    else compute_pair<F, MODE_SLOW>(words, lut_mem, cp, s, z, B, c);
#pragma unroll
                    for (int j = 0; j < 2 * kSets; ++j)
                        if (j == i)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[j >> 1][j & 1][e] += c[e];
                }
            }
            __syncwarp();                                    // every lane has read the stage: it may be filled again
            fetch_weights(stage);
            fetch_x(stage);
            fetch_advance();
            ptx::cp_async_commit();
            if (++stage == D) stage = 0;
        }
        flush(tile);
        seg_lo = seg_end;
    }
    ptx::cp_async_wait_group<0>();
    if (p.om.n_dst > 1) __threadfence_system();              // stores into other GPUs' buffers: before the hand-shake's flag
}

template <int BITS, bool SPARSE, int R>
cudaError_t rows_launch_r(RowsParams p, int sms, int dev, cudaStream_t stream) {
    using F = RFormat<BITS, SPARSE>;
    constexpr int smem = RSmem<F, R>::kBytes;
    auto kern = rows_kernel<BITS, SPARSE, R>;
    static std::atomic<int> ready[16];
    if (ready[dev].load() == 0) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        ready[dev].store(1);
    }
    const int slots = kCtasPerSm * sms;
    p.parts = 1;
    if (p.tiles < slots) {
        int f = slots / p.tiles;
        if (f > p.U / kKLanes) f = p.U / kKLanes;
        if (f > 1) {
            const int rounds = ((p.U + f - 1) / f + kKLanes - 1) / kKLanes;      // steps of the busiest warp
            while (f > 1 && ((p.U + f - 2) / (f - 1) + kKLanes - 1) / kKLanes == rounds) --f;
            p.parts = f;
        }
    }
    const int grid = p.parts > 1 ? p.tiles * p.parts : p.tiles < slots ? p.tiles : slots;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(kRowsThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e == cudaSuccess) count_launch();
    return e;
}

template <int BITS, bool SPARSE>
cudaError_t rows_launch_fmt(const RowsParams& p, int sms, int dev, cudaStream_t stream) {
    if (p.rows == 1) return rows_launch_r<BITS, SPARSE, 1>(p, sms, dev, stream);
    if (p.rows <= 4) return rows_launch_r<BITS, SPARSE, 4>(p, sms, dev, stream);
    return rows_launch_r<BITS, SPARSE, 8>(p, sms, dev, stream);
}

}  // namespace

// Which calls take this kernel by default; every figure is us on one B200, tcgen05 kernel -> this one, calls back to back.
// Alone, its fixed cost per launch is about half of the other's and its rate is lower: one row int4 2048^2 7.7 -> 4.8, 4096 x 12288
// 13.7 -> 13.1, 5120 x 9728 13.7 -> 14.9; int2 5120^2 10.3 -> 9.7.  So the adding route's line is the number of weights.  From more than
// 2 column tiles per SM on, K cannot be cut any more and SMs are left with uneven numbers of tiles: 1024 x 30720 11.5 -> 10.8,
// 1024 x 36864 12.1 -> 10.9, 1024 x 40960 12.7 -> 14.5 (16:32 17.2 -> 17.7).
// A call that overwrites stands between others in a model's layer, and there a change of kernel from one matrix to the next costs
// 2..5 us.  min(N, S) is the layer's width for its every matrix, so a bound on it keeps a layer on one kernel.  Four matrices and
// their row norms, width (inner width), all on the tcgen05 kernel -> those of up to 48 Mi weights (2..8 rows: 16 Mi) on this one:
// one int4 row 5120 (13824) 76.3 -> 76.8, 4096 (11008) 62.5 -> 60.4, 3584 (9472) 54.1 -> 52.4, 3072 (8192) 50.7 -> 43.5, 2048 (5632)
// 42.8 -> 32.0; int2, whose decode is cheapest here, 5120 76.2 -> 74.5, 4096 62.6 -> 55.9.  4 rows int4 4096 66.7 -> 66.2, 3072 53.5 ->
// 52.8, 2560 (6912) 49.2 -> 47.5, 2048 45.5 -> 40.2; 8 rows (larger stages, fewer of them) 3072 55.7 -> 57.9, 2560 51.3 -> 51.0, 2304
// (6144) 49.1 -> 51.4, 2048 49.1 -> 48.6, 1536 (4096) 43.1 -> 39.8.
// Very long columns: the last part adds the sums of hundreds of parts one after the other, 4 rows 65536 x 64 38.8 -> 30.1, 131072 x 64
// 40.9 -> 57.6, 8 rows 32768 x 64 38.0 -> 31.8, 65536 x 64 42.9 -> 58.0.
// The lines were drawn against an older tcgen05 kernel.  Against the present one (its figure first) they hold up to about 8 Mi weights - one row
// int4 2688 x 2432 7.3 -> 5.4, int2 4224 x 1024 6.8 -> 5.3, 4 rows 16:32 4480 x 1344 9.2 -> 6.8 - and lie too far out above: one adding row, alone,
// int4 5120^2 9.5 -> 11.2, int3 9.6 -> 11.8, 16:32 11.1 -> 12.8, 5..8 rows 7680 x 1472 8.8 -> 15.8.  With the zero-fill that an adding row mostly
// follows, and on a first call with new buffers (tensor maps are encoded then), 5120^2 is level or faster here: 11.3 -> 10.8 in a graph, 28.5 -> 26.8.
// (The bounds also keep step and tile numbers far inside 32 bits.)
constexpr long long kMi = 1ll << 20;

bool rows_supported(int bits, bool accumulate, int rows, int N, int S) {
    const long long weights = (long long)N * S;
    const int width = N < S ? N : S;
    if (rows == 1) return weights <= (S > 148 * 2 * kTileCols ? 36 : 48) * kMi && (accumulate || bits == 2 || width <= 3072);
    if (rows < 1 || rows > kMaxRows || weights > 16 * kMi) return false;
    return rows <= 4 ? N <= 131072 && (bits == 2 || width <= 3072) : N <= 65536 && width <= 2560;
}

cudaError_t rows_launch(int bits, bool sparse, const StreamParams& sp, int overlap, cudaStream_t stream) {
    static std::atomic<int> sms_of[16];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    dev &= 15;
    int sms = sms_of[dev].load();
    if (sms == 0) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        sms_of[dev].store(sms);
    }
    RowsParams p{};
    p.om = sp.om;
    p.matrix = sp.matrix;
    p.mask = sp.mask;
    p.x = sp.x;
    p.scales = sp.scales;
    p.zeros = sp.zeros;
    p.partials = reinterpret_cast<unsigned long long*>(sp.partials);
    p.status = sp.status;
    p.rows = sp.rows;
    p.N = sp.N;
    p.S = sp.S;
    p.U = (sp.N + 127) / 128;
    p.tiles = sp.S / kTileCols;
    p.accumulate = sp.accumulate;
    p.overlap = overlap;
    p.gdiv = sp.gdiv;
    if (sparse) return rows_launch_fmt<4, true>(p, sms, dev, stream);
    if (bits == 4) return rows_launch_fmt<4, false>(p, sms, dev, stream);
    if (bits == 3) return rows_launch_fmt<3, false>(p, sms, dev, stream);
    return rows_launch_fmt<2, false>(p, sms, dev, stream);
}

}  // namespace i4mm
