// Row decoders of the tensor-core matvec (vqm_tcmv.cuh): raw words of one row -> A columns, fp16 or bytes.
//
// begin() reads the scales of a unit (half a step of 128 columns, `kh` = which half; scaled bytes: a whole step), chunk<CH>() fills the
// registers of its chunk CH: 32 of 64 fp16 values, 32 of 128 scaled bytes or 16 of 64 signed bytes.  Registers come in core rows of 4
// (8 fp16 columns; 16 bytes); the columns behind them are tc_columns() of the kernel's header.
//   fp16: masked fields are subnormals, field * 2^-24 times the field's place value; the multipliers undo the place value, so every A
//   value is (quant - bias) * sub-scale * 2^-24, exactly (at most 11 significant bits).  scale() is the fp16 super-scale times 2^24.
//   bytes: an A value is an integer, see the second part of this file.  scale() is the super-scale (signed bytes: the scale of 32
//   weights) times tc_piece_unit().
// The comments give the instructions per 8 weights: integer ones go to a pipe that takes a warp instruction every 2 cycles,
// and so does packed fp16 arithmetic, but the two run side by side (measured 1.3 cycles per instruction when mixed).
#pragma once

#include "vqm_tcmv.cuh"

namespace vqm {

constexpr float kTc24 = 16777216.0f;  // 2^24
// Activations as bytes are integers times this and their factor (tc_convert_bytes).
__host__ __device__ constexpr float tc_piece_unit(int type) { return 2.0f / static_cast<float>(1 << tc_piece_bits(type)); }

template <int TYPE>
struct TcUnit;

// Q4_K / Q5_K: d, dmin, 12 bytes of 6-bit scales and minimums; sub-block pairs (low and high nibbles) of 64 columns.
// Q4_K: 5 integer + 4 fp16 instructions per 8 weights.  Q5_K adds the fifth bit with its own multiplier: 11 + 8.
template <int TYPE>
struct TcUnitK45 {
    float d, dm;
    uint32_t sc, mn;  // scales / minimums of the half's four sub-blocks, one per byte
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t line, uint32_t, int kh) {
        const uint4 h = lds128u(line);
        d = half_bits_to_float(h.x & 0xFFFFu) * kTc24;
        dm = half_bits_to_float(h.x >> 16);
        sc = kh == 0 ? h.y & 0x3F3F3F3Fu : (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
        mn = kh == 0 ? h.z & 0x3F3F3F3Fu : ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    }
    __device__ __forceinline__ float scale(int) const { return d; }
    template <int G>
    __device__ __forceinline__ float minimum() const { return dm * byte_to_float<G>(mn); }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t line, uint32_t sh, int kh, uint32_t (&a)[32]) const {
        constexpr uint32_t kNeg1024 = 0xE400E400u, kNeg64 = 0xD400D400u;
        const uint32_t k0 = tc::hadd2(tc::byte_h2<2 * CH>(sc, tc::kHi1024), kNeg1024);    // scale of the low nibbles
        const uint32_t k1 = tc::hadd2(tc::byte_h2<2 * CH + 1>(sc, tc::kHi64), kNeg64);    // of the high ones, / 16
        uint32_t q[8];
        tc::words<TYPE, O, (TYPE == kQ4_K ? 16 : 48) + 32 * CH, 8>(line + 64 * kh, sh, q);
        if constexpr (TYPE == kQ4_K) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t w = q[i], v = w >> 8;
                a[4 * i] = tc::hmul2(w & 0x000F000Fu, k0);
                a[4 * i + 1] = tc::hmul2(w & 0x00F000F0u, k1);
                a[4 * i + 2] = tc::hmul2(v & 0x000F000Fu, k0);
                a[4 * i + 3] = tc::hmul2(v & 0x00F000F0u, k1);
            }
        } else {
            uint32_t f[8];
            tc::words<TYPE, O, 16, 8>(line, sh, f);
            // the fifth bit of sub-block 4 kh + s is bit 4 kh + s of its byte: place value 2^s after the shift, worth 16 * scale
            constexpr uint32_t e0 = (15 + 4 - 2 * CH) << 10, e1 = (15 + 7 - 2 * CH) << 10;  // 2^(4 - s), and 2^(4 - s) * 16 (k1 is / 16)
            const uint32_t f0 = tc::hmul2(k0, e0 * 0x10001u), f1 = tc::hmul2(k1, e1 * 0x10001u);
            constexpr uint32_t m0 = 0x00010001u << (2 * CH), m1 = 0x00010001u << (2 * CH + 1);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t w = q[i], v = w >> 8, b = f[i] >> (4 * kh), c = f[i] >> (4 * kh + 8);
                a[4 * i] = tc::hfma2(w & 0x000F000Fu, k0, tc::hmul2(b & m0, f0));
                a[4 * i + 1] = tc::hfma2(w & 0x00F000F0u, k1, tc::hmul2(b & m1, f1));
                a[4 * i + 2] = tc::hfma2(v & 0x000F000Fu, k0, tc::hmul2(c & m0, f0));
                a[4 * i + 3] = tc::hfma2(v & 0x00F000F0u, k1, tc::hmul2(c & m1, f1));
            }
        }
    }
};
template <>
struct TcUnit<kQ4_K> : TcUnitK45<kQ4_K> {};
template <>
struct TcUnit<kQ5_K> : TcUnitK45<kQ5_K> {};

// Q6_K: low nibbles @0, high bit pairs @128, int8 scales @192, d @208.  Quant times scale needs 14 bits, so a weight is two
// A columns over the same activations: scale * low nibble and 16 * scale * (high bits - 2).  10 + 8 per 8 weights.
// Chunk CH: byte columns 8 CH .. 8 CH + 7 of each of the half's four 32-column quarters.
template <>
struct TcUnit<kQ6_K> {
    float d;
    uint32_t sc[2];  // the half's eight scales (quarter * 2 + half of the quarter), one per byte, + 128
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t line, uint32_t sh, int kh) {
        tc::words<kQ6_K, O, 192, 2>(line + 8 * kh, sh, sc);
        sc[0] ^= 0x80808080u, sc[1] ^= 0x80808080u;
        uint32_t w[1];
        tc::words<kQ6_K, O, 208, 1>(line, sh, w);
        d = half_bits_to_float(w[0] & 0xFFFFu) * kTc24;
    }
    __device__ __forceinline__ float scale(int) const { return d; }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t line, uint32_t sh, int kh, uint32_t (&a)[32]) const {
        constexpr int IS = CH >> 1;
        uint32_t k[4], kh2[4], kb[4];
        {
            const uint32_t n1152 = 0xE480E480u;  // -(1024 + 128)
            k[0] = tc::hadd2(tc::byte_h2<IS>(sc[0], tc::kHi1024), n1152);
            k[1] = tc::hadd2(tc::byte_h2<2 + IS>(sc[0], tc::kHi1024), n1152);
            k[2] = tc::hadd2(tc::byte_h2<IS>(sc[1], tc::kHi1024), n1152);
            k[3] = tc::hadd2(tc::byte_h2<2 + IS>(sc[1], tc::kHi1024), n1152);
#pragma unroll
            for (int i = 0; i < 4; ++i) kb[i] = tc::hmul2(k[i], 0x80208020u);  // * -2^-19: 16 * -2 * 2^-24
            kh2[0] = tc::hmul2(k[0], 0x4C004C00u);                             // 16
            kh2[1] = tc::hmul2(k[1], 0x44004400u);                             // 16 / 4
            kh2[2] = k[2];                                                     // 16 / 16
            kh2[3] = tc::hmul2(k[3], 0x34003400u);                             // 16 / 64
            k[2] = tc::hmul2(k[2], 0x2C002C00u), k[3] = tc::hmul2(k[3], 0x2C002C00u);  // / 16: high nibbles
        }
        uint32_t l0[2], l1[2], hb[2];
        tc::words<kQ6_K, O, 8 * CH, 2>(line + 64 * kh, sh, l0);
        tc::words<kQ6_K, O, 32 + 8 * CH, 2>(line + 64 * kh, sh, l1);
        tc::words<kQ6_K, O, 128 + 8 * CH, 2>(line + 32 * kh, sh, hb);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint32_t *lo = a + 16 * i, *hi = a + 16 * i + 8;
            uint32_t w = l0[i], v = w >> 8;
            lo[0] = tc::hmul2(w & 0x000F000Fu, k[0]);
            lo[1] = tc::hmul2(w & 0x00F000F0u, k[2]);
            lo[2] = tc::hmul2(v & 0x000F000Fu, k[0]);
            lo[3] = tc::hmul2(v & 0x00F000F0u, k[2]);
            w = l1[i], v = w >> 8;
            lo[4] = tc::hmul2(w & 0x000F000Fu, k[1]);
            lo[5] = tc::hmul2(w & 0x00F000F0u, k[3]);
            lo[6] = tc::hmul2(v & 0x000F000Fu, k[1]);
            lo[7] = tc::hmul2(v & 0x00F000F0u, k[3]);
            w = hb[i], v = w >> 8;
            hi[0] = tc::hfma2(w & 0x00030003u, kh2[0], kb[0]);
            hi[1] = tc::hfma2(w & 0x00300030u, kh2[2], kb[2]);
            hi[2] = tc::hfma2(v & 0x00030003u, kh2[0], kb[0]);
            hi[3] = tc::hfma2(v & 0x00300030u, kh2[2], kb[2]);
            hi[4] = tc::hfma2(w & 0x000C000Cu, kh2[1], kb[1]);
            hi[5] = tc::hfma2(w & 0x00C000C0u, kh2[3], kb[3]);
            hi[6] = tc::hfma2(v & 0x000C000Cu, kh2[1], kb[1]);
            hi[7] = tc::hfma2(v & 0x00C000C0u, kh2[3], kb[3]);
        }
    }
};

// ---- bytes ---------------------------------------------------------------------------------------------------------------
// Q3_K and Q2_K: quant times sub-scale fits into 8 bits, so an A column is a byte and ONE 32-bit multiply scales four weights: no
// byte of the product carries into the next.  Half the registers and stores of fp16 and one integer instruction per four weights
// less; a step is one batch.  Bound by unpacking as the others (warp instructions per 8 weights of Q3_K, 1 row: 31.5 as fp16, 21.0 so).
// 17408 x 5120, 1 / 4 / 8 / 16 rows, fp16 and bytes, us: Q3_K 19.8 / 20.9 / 23.0 / 26.6 and 15.3 / 17.3 / 20.4 / 27.0, Q2_K 15.2 / 16.8 /
// 20.6 / 26.6 and 12.2 / 14.4 / 18.1 / 27.2.  Error against 64 bits, Q3_K: 1.5e-7 and 7e-8; with outliers of 1000 times the rest 1e-6 and 7e-8.
// (Q4_K's products need 10 bits, Q6_K's 14: two and three bytes a weight.)
// Chunk CH: byte columns 16 CH .. 16 CH + 15 of each of the eight 32-column groups (half * 4 + j);
// register (half * 4 + i) * 4 + j holds columns 128 half + 32 j + 16 CH + 4 i .. + 3.

// Byte K of `w`, sign-extended.
template <int K>
__device__ __forceinline__ uint32_t tc_signed_byte(uint32_t w) {  // (__byte_perm has no sign replication)
    uint32_t d;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(w), "n"(0x8880 | (K * 0x1111)));
    return d;
}

// Q3_K: high-bit mask @0, bit pairs @32, 12 bytes of 6-bit scales @96, d @108; weight = d * (sc - 32) * (q2 + 4 h - 4).  A byte is
// (sc - 32) * (q2 + 4 h - 4) + 127, 3 .. 255.  6 integer instructions + 3 multiplies per 8 weights.
template <>
struct TcUnit<kQ3_K> {
    float d;
    uint32_t sc[4];  // scales - 32, one per byte: byte 2 (j % 2) + CH of sc[2 half + j / 2]
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t line, uint32_t sh, int) {
        uint32_t s[4];
        tc::words<kQ3_K, O, 96, 4>(line, sh, s);
        d = half_bits_to_float(s[3] & 0xFFFFu) * tc_piece_unit(kQ3_K);
        sc[0] = (s[0] & 0x0F0F0F0Fu) | ((s[2] << 4) & 0x30303030u);
        sc[1] = (s[1] & 0x0F0F0F0Fu) | ((s[2] << 2) & 0x30303030u);
        sc[2] = ((s[0] >> 4) & 0x0F0F0F0Fu) | (s[2] & 0x30303030u);
        sc[3] = ((s[1] >> 4) & 0x0F0F0F0Fu) | ((s[2] >> 2) & 0x30303030u);
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[i] = (sc[i] + 0x60606060u) ^ 0x80808080u;  // (no carries: at most 63 + 96)
    }
    __device__ __forceinline__ float scale(int) const { return d; }
    // Bits 0 and 2 of every byte of `x` at bits 2 and 6 (beside them copies that the caller masks out; a byte stays below 101).
    static __device__ __forceinline__ uint32_t spread(uint32_t x) { return x * 20u; }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t line, uint32_t sh, int, uint32_t (&a)[32]) const {
        uint32_t h[4];
        tc::words<kQ3_K, O, 16 * CH, 4>(line, sh, h);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t k[4], b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t w = sc[2 * half + (j >> 1)];
                k[j] = (j & 1) ? tc_signed_byte<2 + CH>(w) : tc_signed_byte<CH>(w);
                b[j] = 0x7F7F7F7Fu - 0x04040404u * k[j];
            }
            uint32_t q[4];
            if (half == 0) tc::words<kQ3_K, O, 32 + 16 * CH, 4>(line, sh, q);
            else tc::words<kQ3_K, O, 64 + 16 * CH, 4>(line, sh, q);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t m = half == 0 ? h[i] : h[i] >> 4;
                // three-bit quants, one per nibble: groups 0 and 2, groups 1 and 3
                const uint32_t he = spread(m & 0x05050505u), ho = (m & 0x0A0A0A0Au) * 10u;
                const uint32_t e = (q[i] & 0x33333333u) | (he & 0xCCCCCCCCu), o = ((q[i] >> 2) & 0x33333333u) | (ho & 0xCCCCCCCCu);
                uint32_t *r = a + (half * 4 + i) * 4;
                r[0] = (e & 0x07070707u) * k[0] + b[0];
                r[1] = (o & 0x07070707u) * k[1] + b[1];
                r[2] = ((e >> 4) & 0x07070707u) * k[2] + b[2];
                r[3] = ((o >> 4) & 0x07070707u) * k[3] + b[3];
            }
        }
    }
};

// Q2_K: 16 bytes of 4-bit scales and minimums @0, bit pairs @16, d @80, dmin @82.  A byte is 4 * scale * quant, at most 180: the
// upper of two neighbouring bit pairs already has the factor 4.  2.5 integer instructions + 2 multiplies per 8 weights.
template <>
struct TcUnit<kQ2_K> {
    float d, dm;
    uint32_t sc[4], mn[4];  // scales (of even groups times 4) and minimums, one per byte: byte 2 (j % 2) + CH of word 2 half + j / 2
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t line, uint32_t sh, int) {
        uint32_t s[4], w[1];
        tc::words<kQ2_K, O, 0, 4>(line, sh, s);
        tc::words<kQ2_K, O, 80, 1>(line, sh, w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sc[i] = (s[i] & 0x0F0F0000u) | ((s[i] << 2) & 0x00003C3Cu);
            mn[i] = (s[i] >> 4) & 0x0F0F0F0Fu;
        }
        d = half_bits_to_float(w[0] & 0xFFFFu) * (0.25f * tc_piece_unit(kQ2_K));
        dm = half_bits_to_float(w[0] >> 16);
    }
    __device__ __forceinline__ float scale(int) const { return d; }
    template <int G>
    __device__ __forceinline__ float minimum() const { return dm * byte_to_float<G & 3>(mn[G >> 2]); }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t line, uint32_t sh, int, uint32_t (&a)[32]) const {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t q[4];
            if (half == 0) tc::words<kQ2_K, O, 16 + 16 * CH, 4>(line, sh, q);
            else tc::words<kQ2_K, O, 48 + 16 * CH, 4>(line, sh, q);
            const uint32_t k0 = __byte_perm(sc[2 * half], 0u, 0x4440 | CH), k1 = __byte_perm(sc[2 * half], 0u, 0x4442 | CH);
            const uint32_t k2 = __byte_perm(sc[2 * half + 1], 0u, 0x4440 | CH), k3 = __byte_perm(sc[2 * half + 1], 0u, 0x4442 | CH);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t w = q[i], v = w >> 4;
                uint32_t *r = a + (half * 4 + i) * 4;
                r[0] = (w & 0x03030303u) * k0;
                r[1] = (w & 0x0C0C0C0Cu) * k1;
                r[2] = (v & 0x03030303u) * k2;
                r[3] = (v & 0x0C0C0C0Cu) * k3;
            }
        }
    }
};

// N words at any even shared address (the same position within 8 bytes for all lanes): aligned 8-byte loads, one select and
// one funnel shift per word.  For the 34- and 18-byte blocks, whose position changes from block to block.
template <int N>
__device__ __forceinline__ void tc_words_at(uint32_t at, uint32_t (&w)[N]) {
    constexpr int loads = (N + 3) / 2;
    const uint32_t line = at & ~7u, sh = (at & 2u) * 8u;
    const bool upper = (at & 4u) != 0;
    uint32_t r[2 * loads];
#pragma unroll
    for (int i = 0; i < loads; ++i) {
        const unsigned long long v = lds64(line + 8 * i);
        r[2 * i] = static_cast<uint32_t>(v), r[2 * i + 1] = static_cast<uint32_t>(v >> 32);
    }
    uint32_t s[N + 1];
#pragma unroll
    for (int i = 0; i < N + 1; ++i) s[i] = upper ? r[i + 1] : r[i];
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(s[i], s[i + 1], sh);
}

// Q8_0, IQ4_NL, IQ4_XS: the weights (quants, levels) are signed bytes as they are; a scale covers 32 of them, the K of one MMA, and
// multiplies that MMA's sums.  Chunks of 64 weights, 16 registers.  1 / 4 / 8 rows, as fp16 and as bytes, us: IQ4_XS 17408 x 5120 23.4 /
// 25.7 / 31.2 and 18.3 / 23.6 / 31.6; IQ4_NL 5120 x 17408 28.1 / 30.2 / 38.8 and 22.4 / 28.5 / 38.4; Q8_0 17408 x 5120 26.0 / 27.0 / 30.1
// and 23.7 / 24.3 / 29.0 (of which its bytes take 14.5).  Error against 64 bits, IQ4_XS: 1.5e-7 and 7e-8, Q8_0 1.4e-7 and 1.0e-7.
// Q8_0: blocks of 32 int8 behind an fp16 scale.  Nothing to unpack: 4 integer instructions per 8 weights align the words.
template <>
struct TcUnit<kQ8_0> {
    float d[4];  // the half's four blocks
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t, uint32_t, int) {}
    __device__ __forceinline__ float scale(int g) const { return d[g]; }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[16]) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t at = row + 34 * (4 * kh + 2 * CH + g);
            d[2 * CH + g] = half_bits_to_float(lds16(at)) * tc_piece_unit(kQ8_0);
            uint32_t q[8];
            tc_words_at<8>(at + 2, q);
#pragma unroll
            for (int i = 0; i < 8; ++i) a[8 * g + i] = q[i];
        }
    }
};

__device__ __forceinline__ uint32_t tc_prmt(uint32_t a, uint32_t b, uint32_t s) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}
// The 8 nibbles of a word as 8 levels, in the order of the nibbles: the 16 levels of IQ4_NL / IQ4_XS sit in four registers, one per
// byte.  11 integer instructions.
__device__ __forceinline__ void tc_iq4_word(uint32_t w, uint32_t *r) {
    constexpr uint32_t L0 = 0xBFAD9881u, L1 = 0xF6EADDCFu, H0 = 0x26190D01u, H1 = 0x71594535u;
    const uint32_t sel = w & 0x77777777u;                          // entry within each half of the table
    const uint32_t pick = ((w >> 1) & 0x44444444u) | 0x32103210u;  // which half
    r[0] = tc_prmt(tc_prmt(L0, L1, sel), tc_prmt(H0, H1, sel), pick);
    r[1] = tc_prmt(tc_prmt(L0, L1, sel >> 16), tc_prmt(H0, H1, sel >> 16), pick >> 16);
}

// IQ4_NL: blocks of 32 nibbles behind an fp16 scale.
template <>
struct TcUnit<kIQ4_NL> {
    float d[4];
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t, uint32_t, int) {}
    __device__ __forceinline__ float scale(int g) const { return d[g]; }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[16]) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t at = row + 18 * (4 * kh + 2 * CH + g);
            d[2 * CH + g] = half_bits_to_float(lds16(at)) * tc_piece_unit(kIQ4_NL);
            uint32_t q[4];
            tc_words_at<4>(at + 2, q);
#pragma unroll
            for (int i = 0; i < 4; ++i) tc_iq4_word(q[i], a + 8 * g + 2 * i);
        }
    }
};

// IQ4_XS: d @0, high scale bits @2, low scale nibbles @4, nibbles @8; 32-column groups with a 6-bit scale.
template <>
struct TcUnit<kIQ4_XS> {
    float d;
    uint32_t sl, sh6;  // the half's four scale nibbles (16 bits) and bit pairs (8 bits)
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t line, uint32_t, int kh) {
        const unsigned long long h = lds64(line);
        d = half_bits_to_float(static_cast<uint32_t>(h) & 0xFFFFu) * tc_piece_unit(kIQ4_XS);
        sl = static_cast<uint32_t>(h >> 32) >> (16 * kh);
        sh6 = static_cast<uint32_t>(h) >> (16 + 8 * kh);
    }
    __device__ __forceinline__ float scale(int) const { return d; }
    __device__ __forceinline__ int integer_scale(int g) const { return static_cast<int>(((sl >> (4 * g)) & 15u) | (((sh6 >> (2 * g)) & 3u) << 4)) - 32; }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t line, uint32_t sh, int kh, uint32_t (&a)[16]) const {
        uint32_t q[8];
        tc::words<kIQ4_XS, false, 8 + 32 * CH, 8>(line + 64 * kh, sh, q);
#pragma unroll
        for (int i = 0; i < 8; ++i) tc_iq4_word(q[i], a + 2 * i);
    }
};

// ---- codebook types ------------------------------------------------------------------------------------------------------
// Eight weights are magnitude bytes of a codebook in shared memory (one 8-byte or two 4-byte entries), eight sign bits and an
// odd scale 2 s + 1 <= 31; magnitudes are at most 66 (the host checks the codebook), so magnitude * scale is exact in fp16.
// The constant factor (1/8, 1/4 or 1) goes into d.  About 25 instructions per 8 weights: two or three for the index, two masks
// per four magnitudes, one multiply, one shift and one LOP3 for the signs per two.
struct TcGrid {
    float d;
    uint32_t table;  // the codebook
    __device__ __forceinline__ float scale(int) const { return d; }

    // fp16 2 s + 1, twice, from the byte 2 s + 1
    static __device__ __forceinline__ uint32_t odd_scale(uint32_t b) { return tc::hadd2(tc::byte_h2<0>(b, tc::kHi1024), 0xE400E400u); }
    // A core row from two words of magnitudes and the sign byte.  v = signs | signs << 14 puts the signs of weights (i, i + 2)
    // 16 bits apart.  emit7: bit 31 of `eighth` flips weight 7 (types whose eighth sign is implied).
    static __device__ __forceinline__ void emit(uint32_t m0, uint32_t m1, uint32_t signs, uint32_t k, uint32_t *r) {
        const uint32_t v = signs * 0x4001u;
        r[0] = tc::hmul2(m0 & 0x00FF00FFu, k) ^ ((v << 15) & 0x80008000u);
        r[1] = tc::hmul2(__byte_perm(m0, 0u, 0x4341), k) ^ ((v << 14) & 0x80008000u);
        r[2] = tc::hmul2(m1 & 0x00FF00FFu, k) ^ ((v << 11) & 0x80008000u);
        r[3] = tc::hmul2(__byte_perm(m1, 0u, 0x4341), k) ^ ((v << 10) & 0x80008000u);
    }
    static __device__ __forceinline__ void emit7(uint32_t m0, uint32_t m1, uint32_t signs7, uint32_t eighth, uint32_t k, uint32_t *r) {
        emit(m0, m1, signs7, k, r);
        r[3] ^= eighth & 0x80000000u;
    }
    __device__ __forceinline__ void entry8(uint32_t index, uint32_t &m0, uint32_t &m1) const {
        const unsigned long long e = lds64(table + index * 8);
        m0 = static_cast<uint32_t>(e), m1 = static_cast<uint32_t>(e >> 32);
    }
};
template <int K>
__device__ __forceinline__ uint32_t tc_byte(uint32_t w) { return __byte_perm(w, 0u, 0x4440 | K); }
// (everything behind the two bytes of d: the words() offsets of these types count from there)
__device__ __forceinline__ uint32_t tc_line2(uint32_t row) { return (row + 2) & ~3u; }
__device__ __forceinline__ uint32_t tc_shift2(uint32_t row) { return ((row + 2) & 2u) * 8u; }

// IQ2_XS: 32 x (9-bit index, 7 signs) @2, 4-bit scale pairs @66.
template <>
struct TcUnit<kIQ2_XS> : TcGrid {
    uint32_t sc;  // the half's four scale bytes: low nibble for the first 16 weights of 32, high for the others
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t row, uint32_t, int kh) {
        d = half_bits_to_float(lds16(row)) * (kTc24 * 0.125f);
        uint32_t w[1];
        tc::words<kIQ2_XS, false, 64, 1>(tc_line2(row) + 4 * kh, tc_shift2(row), w);
        sc = w[0];
    }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[32]) const {
        uint32_t w[4];
        tc::words<kIQ2_XS, false, 16 * CH, 4>(tc_line2(row) + 32 * kh, tc_shift2(row), w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // two entries, which share a scale
            const uint32_t k = odd_scale(((sc >> (8 * (2 * CH + (i >> 1)) + 4 * (i & 1))) & 15u) * 2u + 1u);
            uint32_t p = (w[i] >> 9) & 0x007F007Fu;
            const uint32_t s = p;
            p ^= p >> 4, p ^= p >> 2, p ^= p >> 1;  // bits 0 and 16: the parities
            uint32_t m0, m1;
            entry8(w[i] & 511u, m0, m1), emit7(m0, m1, s & 127u, p << 31, k, a + 8 * i);
            entry8((w[i] >> 16) & 511u, m0, m1), emit7(m0, m1, s >> 16, p << 15, k, a + 8 * i + 4);
        }
    }
};

// (8-byte loads of the rows: 17408 x 5120, 1 row, 22.1 -> 21.3 us; IQ2_XS, which loads less, loses 1 %, Q2_K 4 %, Q3_K gains nothing.)
// IQ2_S: index low bytes @2, sign bytes @34, index high bits @66, scale pairs @74.
template <>
struct TcUnit<kIQ2_S> : TcGrid {
    uint32_t sc, hi;
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t row, uint32_t, int kh) {
        d = half_bits_to_float(lds16(row)) * (kTc24 * 0.125f);
        uint32_t w[1];
        tc_words_at<1>(row + 2 + 4 * kh + 72, w);
        sc = w[0];
        tc_words_at<1>(row + 2 + 4 * kh + 64, w);
        hi = w[0];
    }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[32]) const {
        uint32_t w[2], s[2];
        tc_words_at<2>(row + 2 + 16 * kh + 8 * CH, w);
        tc_words_at<2>(row + 2 + 16 * kh + 32 + 8 * CH, s);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t b = sc >> (8 * (2 * CH + g)), q = hi >> (8 * (2 * CH + g));
            const uint32_t k0 = odd_scale((b & 15u) * 2u + 1u), k1 = odd_scale(((b >> 4) & 15u) * 2u + 1u);
            uint32_t m0, m1;
            uint32_t *r = a + 16 * g;
            entry8(tc_byte<0>(w[g]) | ((q << 8) & 0x300u), m0, m1), emit(m0, m1, tc_byte<0>(s[g]), k0, r);
            entry8(tc_byte<1>(w[g]) | ((q << 6) & 0x300u), m0, m1), emit(m0, m1, tc_byte<1>(s[g]), k0, r + 4);
            entry8(tc_byte<2>(w[g]) | ((q << 4) & 0x300u), m0, m1), emit(m0, m1, tc_byte<2>(s[g]), k1, r + 8);
            entry8(tc_byte<3>(w[g]) | ((q << 2) & 0x300u), m0, m1), emit(m0, m1, tc_byte<3>(s[g]), k1, r + 12);
        }
    }
};

// ---- codebook types with a signed table ---------------------------------------------------------------------------------------
// IQ2_XXS, IQ3_XXS, IQ3_S: the codebook lies in shared memory with every combination of four signs applied, as bytes weight + 128, so ONE
// permute makes the index of four weights out of its index byte and a byte with their signs (and a ninth index bit, or which half of an
// 8-weight entry):
//   word idx + 256 * (signs + 16 * upper) of the table
// A byte masked out is an fp16 subnormal, and one FMA takes the 128 out and applies the scale, exactly.  8 to 11 integer instructions + 4 FMAs
// per 8 weights.  What bounds them then is shared memory (80 % busy before): random words of a table conflict (see tc_table_copies), and
// 4-byte loads of the rows take four turns for 128 bytes where 8-byte ones take four for 256 and a select per word.  IQ3_S, IQ3_XXS, IQ2_XXS
// 17408 x 5120, 1 row, us: masks and shifts for the signs 24.6 / 23.2 / 20.3, signed table 23.9 / 22.4 / 20.1, 8-byte loads 22.3 / 20.9 / 19.4,
// copies of the table 21.8 / 20.1 / 18.8.  (As signed bytes with a sum per 32 columns, like Q8_0: 22.8 / 21.5 / 18.9 with 1 row, but 31.6 / 29.9 / 28.0
// with 8 and twice that with 16, where these take 26.0 / 23.7 / 22.2 and 31.2 / 27.5 / 27.5.)
template <int TYPE, int MC>
__device__ __forceinline__ void tc_make_signed_table(const uint8_t *codebook, uint32_t table) {  // the decoder threads
    constexpr int kWords = TYPE == kIQ3_XXS ? 256 : 512, kSigns = 16 * kWords / kTcDecoders;
    const int word = threadIdx.x % kWords, sign0 = threadIdx.x / kWords * kSigns, idx = word & 255, upper = word >> 8;
    const uint32_t m = reinterpret_cast<const uint32_t *>(codebook)[TYPE == kIQ2_XXS ? 2 * idx + upper : word];
#pragma unroll
    for (int i = 0; i < kSigns; ++i) {
        const uint32_t s = static_cast<uint32_t>(sign0 + i), neg = (s * 0x00204081u) & 0x01010101u;
        const uint32_t v = ((m ^ (neg * 0x7Fu)) + neg) ^ (neg << 7) ^ 0x80808080u;  // (magnitudes below 128; no carries, a zero stays one)
        constexpr int kCopies = tc_table_copies(TYPE, MC);
        const uint32_t at = table + (idx + 256 * (static_cast<int>(s) + 16 * upper)) * (4 * kCopies);
        if constexpr (kCopies == 1) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
        else if constexpr (kCopies == 2) asm volatile("st.shared.v2.u32 [%0], {%1, %1};" ::"r"(at), "r"(v) : "memory");
        else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(v) : "memory");
    }
}
struct TcSigned {
    float d;
    uint32_t table, pitch;  // this lane's copy, and bytes from a word of it to the next
    __device__ __forceinline__ float scale(int) const { return d; }
    // what an entry's bytes are multiplied by, and what is added: k and -128 k, times 2^-24 both
    struct Scale {
        uint32_t k, b;
        __device__ __forceinline__ explicit Scale(uint32_t odd) : k(TcGrid::odd_scale(odd)), b(tc::hmul2(k, 0x80808080u)) {}
    };
    // half a core row: the four weights of index byte I of `idx`, signs and upper bit in byte S of `signs`
    template <int I, int S>
    __device__ __forceinline__ void entry(uint32_t idx, uint32_t signs, const Scale &s, uint32_t *r) const {
        uint32_t at;  // (bytes 2 and 3: the sign of `signs`' byte, which is below 32)
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(at) : "r"(idx), "r"(signs), "n"(I | (4 + S) << 4 | (12 + S) << 8 | (12 + S) << 12));
        const uint32_t w = lds32(table + at * pitch);
        r[0] = tc::hfma2(w & 0x00FF00FFu, s.k, s.b);
        r[1] = tc::hfma2(__byte_perm(w, 0u, 0x4341), s.k, s.b);
    }
    // Four 7-bit fields, each into a byte with its parity on top: the signs of 8 weights, of which the eighth is implied.
    static __device__ __forceinline__ uint32_t signs8(uint32_t aux) {
        const uint32_t y = (aux & 0x7Fu) | ((aux << 1) & 0x7F00u) | ((aux << 2) & 0x7F0000u) | ((aux << 3) & 0x7F000000u);
        uint32_t p = y ^ (y >> 4);
        p ^= p >> 2;
        p ^= p >> 1;
        return y | ((p << 7) & 0x80808080u);
    }
};

// IQ2_XXS: per 32 weights four index bytes and a word of 4 x 7 signs and a 4-bit scale.
template <>
struct TcUnit<kIQ2_XXS> : TcSigned {
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t row, uint32_t, int) { d = half_bits_to_float(lds16(row)) * (kTc24 * 0.125f); }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[32]) const {
        uint32_t w[4];
        tc_words_at<4>(row + 2 + 32 * kh + 16 * CH, w);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t idx = w[2 * g], y = signs8(w[2 * g + 1]), lo = y & 0x0F0F0F0Fu, hi = ((y >> 4) & 0x0F0F0F0Fu) | 0x10101010u;
            const Scale k((w[2 * g + 1] >> 27) | 1u);
            uint32_t *r = a + 16 * g;
            entry<0, 0>(idx, lo, k, r), entry<0, 0>(idx, hi, k, r + 2), entry<1, 1>(idx, lo, k, r + 4), entry<1, 1>(idx, hi, k, r + 6);
            entry<2, 2>(idx, lo, k, r + 8), entry<2, 2>(idx, hi, k, r + 10), entry<3, 3>(idx, lo, k, r + 12), entry<3, 3>(idx, hi, k, r + 14);
        }
    }
};

// IQ3_XXS: two index bytes per 8 weights @2, per 32 weights a word of 4 x 7 signs and a 4-bit scale @66.
template <>
struct TcUnit<kIQ3_XXS> : TcSigned {
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t row, uint32_t, int) { d = half_bits_to_float(lds16(row)) * (kTc24 * 0.25f); }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[32]) const {
        uint32_t w[4], x[2];
        tc_words_at<4>(row + 2 + 32 * kh + 16 * CH, w);
        tc_words_at<2>(row + 2 + 16 * kh + 64 + 8 * CH, x);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t i0 = w[2 * g], i1 = w[2 * g + 1], y = signs8(x[g]), lo = y & 0x0F0F0F0Fu, hi = (y >> 4) & 0x0F0F0F0Fu;
            const Scale k((x[g] >> 27) | 1u);
            uint32_t *r = a + 16 * g;
            entry<0, 0>(i0, lo, k, r), entry<1, 0>(i0, hi, k, r + 2), entry<2, 1>(i0, lo, k, r + 4), entry<3, 1>(i0, hi, k, r + 6);
            entry<0, 2>(i1, lo, k, r + 8), entry<1, 2>(i1, hi, k, r + 10), entry<2, 3>(i1, lo, k, r + 12), entry<3, 3>(i1, hi, k, r + 14);
        }
    }
};

// IQ3_S: index low bytes @2, index high bits @66, sign bytes @74, 4-bit scales @106.
template <>
struct TcUnit<kIQ3_S> : TcSigned {
    uint32_t sc, hi;
    template <bool O>
    __device__ __forceinline__ void begin(uint32_t row, uint32_t, int kh) {
        d = half_bits_to_float(lds16(row)) * kTc24;
        uint32_t w[1];
        tc_words_at<1>(row + 2 + 104, w);
        sc = w[0] >> (16 * kh);
        tc_words_at<1>(row + 2 + 4 * kh + 64, w);
        hi = w[0];
    }
    template <bool O, int CH>
    __device__ __forceinline__ void chunk(uint32_t row, uint32_t, int kh, uint32_t (&a)[32]) const {
        uint32_t w[4], s[2];
        tc_words_at<4>(row + 2 + 32 * kh + 16 * CH, w);
        tc_words_at<2>(row + 2 + 16 * kh + 72 + 8 * CH, s);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t q = hi >> (8 * (2 * CH + g)), i0 = w[2 * g], i1 = w[2 * g + 1];
            // the high bits of the even and of the odd entries, at bit 4 of the bytes of their signs (a multiply spreads them: bit 2 k goes to
            // 8 k + 4; what the other products leave lies elsewhere, and carries stay on odd bits)
            const uint32_t even = (s[g] & 0x0F0F0F0Fu) | (((q & 0x55u) * 0x00410410u) & 0x10101010u);
            const uint32_t odd = ((s[g] >> 4) & 0x0F0F0F0Fu) | (((q & 0xAAu) * 0x00208208u) & 0x10101010u);
            const Scale k(((sc >> (4 * (2 * CH + g))) & 15u) * 2u + 1u);
            uint32_t *r = a + 16 * g;
            entry<0, 0>(i0, even, k, r), entry<1, 0>(i0, odd, k, r + 2), entry<2, 1>(i0, even, k, r + 4), entry<3, 1>(i0, odd, k, r + 6);
            entry<0, 2>(i1, even, k, r + 8), entry<1, 2>(i1, odd, k, r + 10), entry<2, 3>(i1, even, k, r + 12), entry<3, 3>(i1, odd, k, r + 14);
        }
    }
};

}  // namespace vqm
