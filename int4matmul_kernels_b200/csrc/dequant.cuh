// Dequantisation arithmetic shared by the kernels: packed fields planted into fp16 mantissas, then the reference's two
// fp16 roundings (matmul.cuh:115-125) or, per weight, either coding.
#pragma once

#include "common.cuh"

namespace i4mm {

// MODE_WIDE: 16:32 only, the fast mode for zero-points up to 255.  MODE_SLOW, MODE_EITHER: either coding by the column, the first by conversions, weight
// by weight.
enum : int { MODE_FAST = 0, MODE_GENERAL = 1, MODE_SLOW = 2, MODE_WIDE = 3, MODE_EITHER = 4 };

// (mask & a) | (~mask & b)
__device__ __forceinline__ uint32_t bit_select(uint32_t mask, uint32_t a, uint32_t b) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(d) : "r"(mask), "r"(a), "r"(b));
    return d;
}
// (a & b) ^ c
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// ---- per-column constants ---------------------------------------------------------------------------------
struct ColK {
    uint32_t s2, z2;
    uint32_t zb;       // sparse fast mode: the integer zero-point replicated into 4 bytes
};

// v = (1024 + q_lo * 2^a, 1024 + q_hi * 2^b) -> the two fp16 weights.  mul / base undo the two shifts exactly.
template <int BITS, int MODE>
__device__ __forceinline__ uint32_t finish(uint32_t v, uint32_t mul, uint32_t base, uint32_t off, const ColK& c) {
    if (MODE == MODE_FAST || MODE == MODE_WIDE) return hmul2_u(hfma2_u(v, mul, off), c.s2);         // off = base - zero
    const uint32_t q = hfma2_u(v, mul, base);                                  // exact integers
    if (MODE == MODE_GENERAL) return hmul2_u(hsub2_u(q, c.z2), c.s2);
    if (MODE == MODE_EITHER) {
        // dequant_dynamic for both halves, +-2^(q & EXP) put together from its bits
        constexpr uint32_t SGN = 0x10001u << (BITS - 1), EXP = SGN - 0x10001u;
        const uint32_t qi = hadd2_u(q, kMagic1024);                            // q in the low bits
        const uint32_t power = (((qi & EXP) << 10) + 0x3C003C00u) | ((qi & SGN) << (16 - BITS));
        const uint32_t lin = hmul2_u(hsub2_u(q, c.z2), c.s2), expo = hfma2_u(power, c.s2 ^ 0x80008000u, c.z2);
        return __hge(__ushort_as_half((unsigned short)(c.s2 & 0xFFFFu)), __ushort_as_half(0)) ? lin : expo;
    }
    const __half2 qh = u32_as_h2(q);
    const __half s = __ushort_as_half((unsigned short)(c.s2 & 0xFFFFu));
    const __half z = __ushort_as_half((unsigned short)(c.z2 & 0xFFFFu));
    const __half lo = dequant_dynamic<BITS>(__half2uint_rz(__low2half(qh)), s, z);
    const __half hi = dequant_dynamic<BITS>(__half2uint_rz(__high2half(qh)), s, z);
    return h2_as_u32(__halves2half2(lo, hi));
}

// half2 constants (hi << 16 | lo)
constexpr uint32_t MUL_1_16 = 0x2C003C00u, BASE_1_16 = 0xD400E400u;      // (x1, x16): int4 nibble pairs
constexpr uint32_t MUL_1_4 = 0x34003C00u, BASE_1_4 = 0xDC00E400u;        // (x1, x4):  int2 crumbs 0, 1
constexpr uint32_t MUL_16_64 = 0x24002C00u, BASE_16_64 = 0xCC00D400u;    // (x16, x64): int2 crumbs 2, 3
constexpr uint32_t MUL_1_8 = 0x30003C00u, BASE_1_8 = 0xD800E400u;        // (x1, x8):  int3 field pairs
constexpr uint32_t MUL_1_1 = 0x3C003C00u, BASE_1_1 = 0xE400E400u;        // (x1, x1): sparse int4 through bytes

// ---- 16:32 sparse: the next 8 positions of a 32-block ---------------------------------------------------------------
// The next 8 kept nibbles are spread over the bytes of a register pair (even nibbles, odd nibbles); two PRMTs put them
// at their positions.  The selectors of both PRMTs are one 32-bit word of a 256-entry table indexed by the byte of the
// keep-mask (nibble j of the word belongs to position j).  A dropped position selects 8, for which PRMT replicates the
// sign of a byte below 128 (a nibble, XORed with a zero-point below 128): it yields 0x00.  A 1 KB table: the same look-up in a
// table of 16-byte entries (selectors, masks and popcount) takes ~10 shared-memory wavefronts per warp instead of ~3.5, because
// random entries of four banks collide.
constexpr int kSparseLutEntries = 256;
__device__ __forceinline__ uint32_t sparse_selectors(int keep) {
    uint32_t sel = 0, rank = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        uint32_t s = 8;
        if (keep & (1 << j)) {
            s = (rank >> 1) + 4u * (rank & 1u);
            ++rank;
        }
        sel |= s << (4 * j);
    }
    return sel;
}

// A <- the four pairs of byte `step` (0..3, in this order) of keep-mask m; (hi : lo) is the stream of kept nibbles.
template <int MODE>
__device__ __forceinline__ void sparse_expand(uint32_t& lo, uint32_t& hi, uint32_t m, int step, const uint32_t* lut, const ColK& c,
                                              uint32_t (&A)[4]) {
    const uint32_t byte4 = (step == 0 ? m << 2 : m >> (8 * step - 2)) & 0x3FCu;          // 4 x the mask byte: table offset
    const uint32_t sel = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(lut) + byte4);
    // Fast mode: a dropped position gets the (integer) zero-point as its nibble, so it decodes to +0.  The nibbles go through
    // the PRMT with the zero-point XORed in, which the extraction's LOP3 does for nothing, so that a dropped position's 0x00 and
    // a kept one's nibble both come right by one XOR afterwards (a mask of the kept positions and a select were two
    // instructions of five per 4 positions: one row 16384 x 16384 57.3 -> 54.4 us, 2048 rows 5120 x 20480 350.5 -> 340.4; few-row
    // kernel 2048 x 5632 1 row 8.4 -> 8.1, 8 rows 11.6 -> 11.4, of 24 sizes only 2048 x 2048 with 5..8 rows is slower, 8.0 -> 8.1)
    const uint32_t flip = MODE == MODE_FAST ? c.zb : 0u;
    uint32_t even = and_xor(lo, 0x0F0F0F0Fu, flip), odd = and_xor(lo >> 4, 0x0F0F0F0Fu, flip), pick = sel;
    const uint32_t off = hsub2_u(BASE_1_1, c.z2);
    if (MODE == MODE_WIDE) {
        // No XOR brings both a kept byte (below 128) and a dropped one right here.  But where a position is dropped, the eighth nibble is not
        // used: the zero-point takes its place, and dropped positions select it instead of 8.
        odd = prmt(odd, c.zb, byte4 == 0x3FCu ? 0x3210u : 0x4210u);
        pick = sel - ((sel >> 3) & 0x11111111u);
    }
#pragma unroll
    for (int q4 = 0; q4 < 2; ++q4) {
        const uint32_t s = q4 ? pick >> 16 : pick;                                       // (PRMT reads the low 16 bits)
        const uint32_t d = prmt(even, odd, s) ^ flip;
        A[2 * q4] = finish<4, MODE>(prmt(d, 0x64646464u, 0x5140), MUL_1_1, BASE_1_1, off, c);
        A[2 * q4 + 1] = finish<4, MODE>(prmt(d, 0x64646464u, 0x7362), MUL_1_1, BASE_1_1, off, c);
        if (MODE != MODE_FAST && MODE != MODE_WIDE) {                                    // exact zeros at dropped positions
            const uint32_t k = prmt(0x7F7F7F7Fu, 0x7F7F7F7Fu, s) << 1;                   // kept 0xFE, dropped 0x00: the sign says which
            A[2 * q4] &= prmt(k, k, 0x9988);
            A[2 * q4 + 1] &= prmt(k, k, 0xBBAA);
        }
    }
    const uint32_t used = 4u * (uint32_t)__popc(byte4);                                  // bits of the stream, up to 32
    lo = __funnelshift_rc(lo, hi, used);
    hi = __funnelshift_rc(hi, 0u, used);
}

}  // namespace i4mm
