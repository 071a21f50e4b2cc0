// The kernel of the tensor-core matvec; vqm_tcmv.cuh has the description.
#pragma once

#include "vqm_tcmv_decoders.cuh"

namespace vqm {

template <int N>
struct TcInt {
    static constexpr int value = N;
};

// First columns of the two 4-column words a and b whose 8 columns make core row `l` (0..31) of a step's B operand.
template <int TYPE>
__device__ __forceinline__ void tc_columns(int l, int &a, int &b) {
    if constexpr (TYPE == kQ4_K || TYPE == kQ5_K) {  // chunk of 64 columns, word of its 32 bytes
        a = 64 * (l >> 3) + 4 * (l & 7), b = a + 32;
    } else if constexpr (TYPE == kQ6_K) {            // half, word, pair of quarters
        a = 128 * (l >> 4) + 32 * (l & 1) + 4 * ((l >> 1) & 7), b = a + 64;
    } else if constexpr (tc_scaled_bytes(TYPE)) {    // (half a row of 16 columns) chunk, half, word, pair of 32-column groups
        a = 128 * ((l >> 3) & 1) + 16 * (l >> 4) + 4 * ((l >> 1) & 3) + 64 * (l & 1), b = a + 32;
    } else if constexpr (TYPE == kIQ4_NL || TYPE == kIQ4_XS) {
        a = 32 * (l >> 2) + 4 * (l & 3), b = a + 16;
    } else {
        a = 8 * l, b = a + 4;
    }
}

// The B operand of bytes: six planes.  x = 2^(e - 126 - T) (p0 + 2^-15 p1 + 2^-30 p2), e the biased exponent of the largest magnitude of the
// chunk (`big`), the pieces integers, p0 of at most 2^T (T = tc_piece_bits: 14 or 11), p1 and p2 of at most 2^14: each the rest of the one
// before it, rounded to nearest.  An activation down to 2^-(T + 6) of the largest loses nothing, a smaller one at most 2^-(T + 30) of the
// largest.  (Four planes of one 32-bit integer, 2^-31 of the largest: an output row whose weight is zero at an activation of 10^5 times the
// rest was off by 2e-5 of its own products, now by 1e-7, as with three planes of fp16.)
// Planes 2 q and 2 q + 1 are the upper and the lower byte of p_q: unsigned ones of p_q + 2^15, and one row of ones behind them gives the sum
// of A that 2^15 is taken out with; signed ones its digits, -128 .. 127.  Sums of products are integers and exact.
//   v: the lane's 2 x 4 columns (tc_columns), half a core row.  info: [rows] factors 2^(e - 127); with an offset of A's bytes, then: the
//   three integers -offset * sum of p_q.
template <int TYPE, int MC, bool ONES>
__device__ __forceinline__ void tc_convert_bytes(float (&v)[8], uint32_t big, int t, uint32_t b_stage, uint32_t info, int lane) {
    constexpr bool kSigned = !tc_scaled_bytes(TYPE);
    constexpr unsigned kOffset = tc_byte_offset(TYPE);
    const uint32_t e = big > 1u ? big : 1u;
    // 2^(126 + T - e), in two factors where the power is beyond fp32
    constexpr uint32_t kTop = tc_piece_bits(TYPE);
    const float up = __uint_as_float((e < kTop - 1u ? 254u : 253u + kTop - e) << 23);
    if (e < kTop - 1u) {
        const float up2 = __uint_as_float((126u + kTop - e) << 23);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= up2;
    }
    constexpr int order[2][8] = {{0, 1, 2, 3, 4, 5, 6, 7}, {0, 4, 1, 5, 2, 6, 3, 7}};  // (IQ4: low and high nibbles in turn)
    constexpr int kOrder = tc_order(TYPE) == kOrderBytes ? 1 : 0;
    // added to a number below 2^15, this leaves its nearest integer in the low bits, and what is added to a piece for its bytes' sake
    constexpr float kRound = 12582912.0f + (kSigned ? 128.0f : 32768.0f);
    const f32x2 round = pack2(kRound, kRound), minus = pack2(-1.0f, -1.0f), next = pack2(32768.0f, 32768.0f), up_2 = pack2(up, up);
    const uint32_t at = b_stage + (lane >> 1) * kTcCore + (lane & 1) * 8;
    f32x2 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = mul2(pack2(v[order[kOrder][2 * i]], v[order[kOrder][2 * i + 1]]), up_2);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        uint32_t x[8], plane[2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f32x2 n = add2(r[i], round);
            if (q < 2) r[i] = mul2(add2(r[i], fma2(n, minus, round)), next);  // the rest, exactly
            float lo, hi;
            unpack2(n, lo, hi);
            x[2 * i] = __float_as_uint(lo), x[2 * i + 1] = __float_as_uint(hi);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const uint32_t *c = x + 4 * w;
            const uint32_t c01 = __byte_perm(c[0], c[1], 0x5140), c23 = __byte_perm(c[2], c[3], 0x5140);
            plane[0][w] = __byte_perm(c01, c23, 0x7632), plane[1][w] = __byte_perm(c01, c23, 0x5410);
            if constexpr (kSigned) plane[1][w] ^= 0x80808080u;
        }
        if constexpr (kOffset != 0) {
            unsigned sum[2];
#pragma unroll
            for (int p = 0; p < 2; ++p) sum[p] = __dp4a(plane[p][0], 0x01010101u, __dp4a(plane[p][1], 0x01010101u, 0u));
            const unsigned all = __reduce_add_sync(0xFFFFFFFFu, 256u * sum[0] + sum[1]);  // of p_q + 2^15
            if (lane == 0)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(info + ((q + 1) * tc_info_rows(MC) + t) * 4), "r"(kOffset * (32768u * kTcStepCols - all)) : "memory");
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int n = (2 * q + p) * MC + t;
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + (n >> 3) * tc_group_b(TYPE) + (n & 7) * 16), "r"(plane[p][0]), "r"(plane[p][1]) : "memory");
        }
    }
    if (lane == 0) {
        // an infinite or undefined activation makes the outputs undefined: they are worked out again (tc_plain_sum)
        const float down = big == 255u ? __uint_as_float(0x7FC00000u) : __uint_as_float(e << 23);
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(info + t * 4), "f"(down) : "memory");
    }
    if (tc_ones_row(TYPE, MC) && ONES && t == 0) {
        constexpr int n = kTcPlanes * MC;
        asm volatile("st.shared.v2.u32 [%0], {%1, %1};" ::"r"(at + (n >> 3) * tc_group_b(TYPE) + (n & 7) * 16), "r"(0x01010101u) : "memory");
    }
}

// The B operand of fp16: three planes, x = s * (h0 + 2^-11 h1 + 2^-22 h2), s a power of two that brings the largest magnitude below 2^10
// (`big`: its biased exponent).
//   v: the lane's 2 x 4 columns, a core row; info: [rows] factors
template <int TYPE, int MC>
__device__ __forceinline__ void tc_convert_halves(const float (&v)[8], uint32_t big, int t, uint32_t b_stage, uint32_t info, int lane) {
    const uint32_t want = 263u - big, e = want < 253u ? want : 253u;
    const float up = __uint_as_float(e << 23);
    if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(info + t * 4), "f"(__uint_as_float((254u - e) << 23)) : "memory");
    constexpr int kOrder = tc_order(TYPE);
    constexpr int order[3][8] = {{0, 2, 4, 6, 1, 3, 5, 7}, {0, 1, 4, 5, 2, 3, 6, 7}, {0, 2, 1, 3, 4, 6, 5, 7}};
    uint32_t h[3][4];
    const f32x2 up2 = pack2(up, up), k2048 = pack2(2048.0f, 2048.0f), neg = pack2(-2048.0f, -2048.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f32x2 r = mul2(pack2(v[order[kOrder][2 * i]], v[order[kOrder][2 * i + 1]]), up2);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            float lo, hi;
            unpack2(r, lo, hi);
            asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h[p][i]) : "f"(hi), "f"(lo));
            if (p < 2) {  // 2048 * (r - plane), exactly
                const float flo = half_bits_to_float(h[p][i] & 0xFFFFu), fhi = half_bits_to_float(h[p][i] >> 16);
                r = fma2(pack2(flo, fhi), neg, mul2(r, k2048));
            }
        }
    }
    const uint32_t at = b_stage + lane * kTcCore;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int n = p * MC + t;
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + (n >> 3) * tc_group_b(TYPE) + (n & 7) * 16), "r"(h[p][0]), "r"(h[p][1]),
                     "r"(h[p][2]), "r"(h[p][3])
                     : "memory");
    }
}

// A lane's 2 x 4 columns (tc_columns) of a row of activations (or of what the fused prologues need beside them): v[0..3] and v[4..7].
struct TcColumns {
    float v[8];
    template <bool CG>
    __device__ __forceinline__ void load(const float *from, int ca, int cb, bool has_a, bool has_b) {
        const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 *pa = reinterpret_cast<const float4 *>(from + ca), *pb = reinterpret_cast<const float4 *>(from + cb);
        const float4 xa = has_a ? (CG ? __ldcg(pa) : *pa) : z, xb = has_b ? (CG ? __ldcg(pb) : *pb) : z;
        v[0] = xa.x, v[1] = xa.y, v[2] = xa.z, v[3] = xa.w, v[4] = xb.x, v[5] = xb.y, v[6] = xb.z, v[7] = xb.w;
    }
};
// Activation row t in the step at col0, before the loop.  cols_here: how many columns exist (a multiple of 32: a word exists as a whole)
template <int TYPE>
__device__ __forceinline__ void tc_fetch(const MatvecArgs &args, int t, int col0, int cols_here, int lane, TcColumns &c) {
    int ca, cb;
    tc_columns<TYPE>(lane, ca, cb);
    const bool has_a = ca < cols_here, has_b = cb < cols_here;
    const size_t at = static_cast<size_t>(t) * args.cols + col0;
    c.load<true>(args.x + at, ca, cb, has_a, has_b);
    if (args.fuse & (kFuseSiluMul | kFuseNorm)) {  // requested now, used by tc_convert
        auto prefetch = [&](const float *from) {
            if (has_a) asm volatile("prefetch.global.L1 [%0];" ::"l"(from + ca));
            if (has_b) asm volatile("prefetch.global.L1 [%0];" ::"l"(from + cb));
        };
        if (args.fuse & kFuseSiluMul) prefetch(args.x2 + at);
        if (args.fuse & kFuseNorm) prefetch(args.norm_w + col0);
    }
}

// Converts activation row t's 256 columns of a step into the B operand: called by a whole warp, lane = core row (bytes: half of one).
//   c: the lane's columns; info: where the row's scale and group sums go (floats [MC] scales, padded to 4, then [groups][MC]); norm_part:
//   where the row's sum of squares goes (0: nowhere); ONES: before the loop, when bytes want their row of ones
template <int TYPE, int MC, bool ONES>
__device__ __forceinline__ void tc_convert(const MatvecArgs &args, TcColumns &c, int t, int col0, int cols_here, uint32_t b_stage, uint32_t info,
                                           uint32_t norm_part, int lane) {
    float (&v)[8] = c.v;
    if (args.fuse & (kFuseSiluMul | kFuseNorm)) {
        int ca, cb;
        tc_columns<TYPE>(lane, ca, cb);
        const bool has_a = ca < cols_here, has_b = cb < cols_here;
        if (args.fuse & kFuseSiluMul) {
            TcColumns g;
            g.load<false>(args.x2 + static_cast<size_t>(t) * args.cols + col0, ca, cb, has_a, has_b);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = v[i] / (1.0f + expf(-v[i])) * g.v[i];
        }
        if (args.fuse & kFuseNorm) {
            // the rms factor of a row is linear: it multiplies the finished outputs, here only the squares are added up
            float sq = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) sq = fmaf(v[i], v[i], sq);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, off);
            if (lane == 0 && norm_part != 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(norm_part), "f"(sq) : "memory");
            TcColumns w;
            w.load<false>(args.norm_w + col0, ca, cb, has_a, has_b);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] *= w.v[i];
        }
    }
    if constexpr (tc_mins(TYPE) > 0) {
        // sums of the columns that share a minimum, for the a and the b words: 8 lanes (32 columns) or 4 lanes (16)
        float sa = (v[0] + v[1]) + (v[2] + v[3]), sb = (v[4] + v[5]) + (v[6] + v[7]);
        constexpr bool k32 = TYPE != kQ2_K;
#pragma unroll
        for (int off = 4; off >= (k32 ? 1 : 2); off >>= 1) {
            sa += __shfl_xor_sync(0xFFFFFFFFu, sa, off);
            sb += __shfl_xor_sync(0xFFFFFFFFu, sb, off);
        }
        // group of a: sub-block 2 c (Q4_K, Q5_K), or 8 half + 2 j + chunk with j = 2 * (lane & 1) (Q2_K); b: the one after / two after
        const bool writer = k32 ? (lane & 7) == 0 : (lane & 6) == 0;
        const int ga = k32 ? 2 * (lane >> 3) : 8 * ((lane >> 3) & 1) + 4 * (lane & 1) + (lane >> 4), gb = ga + (k32 ? 1 : 2);
        if (writer) {
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(info + (tc_info_scales(TYPE, MC) + ga * MC + t) * 4), "f"(sa) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(info + (tc_info_scales(TYPE, MC) + gb * MC + t) * 4), "f"(sb) : "memory");
        }
    }
    uint32_t big = 0;  // the largest magnitude's bits, shifted left by the sign
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const uint32_t m0 = __float_as_uint(v[i]) * 2u, m1 = __float_as_uint(v[i + 1]) * 2u;
        big = max(big, max(m0, m1));
    }
    big = __reduce_max_sync(0xFFFFFFFFu, big) >> 24;
    if constexpr (tc_bytes(TYPE)) tc_convert_bytes<TYPE, MC, ONES>(v, big, t, b_stage, info, lane);
    else tc_convert_halves<TYPE, MC>(v, big, t, b_stage, info, lane);
}

// A unit is what a group of warps takes of a step: one or two halves of 128 columns.  Its chunks go to the tensor cores in
// batches; tensor memory holds one batch of a group and its sums, 128 columns in all.  Types with a scale per 32 columns have a sum
// per 32 columns: from N = 32 on only one chunk's fit.
// Scaled bytes: a unit is a whole step, of two chunks.
__host__ __device__ constexpr int tc_halves(int type) { return tc_wide(type) && !tc_scaled_bytes(type) ? 2 : 1; }
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_batch_chunks() { return (tc_block32(TYPE) && MC > 2) || (tc_scaled_bytes(TYPE) && MC > 8) || MC > 16 ? 1 : 2; }
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_half_batches() { return 2 * tc_parts(TYPE) / tc_batch_chunks<TYPE, MC>(); }
// sums per row that a batch leaves
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_sums() { return tc_block32(TYPE) ? 2 * tc_batch_chunks<TYPE, MC>() : 1; }
// whether a batch starts new sums (else only a unit's first one does)
__host__ __device__ constexpr bool tc_fresh_batches(int type) { return tc_block32(type); }

// What sums have to be multiplied with when they come back from tensor memory, one batch later.
template <int TYPE, int MC>
struct TcPending {
    float s[tc_sums<TYPE, MC>()];        // scales of the sums (their bits are integers where tc_integer_scale)
    float d;                             // the unit's super-scale then
    uint32_t ones;                       // the sum of a unit's A bytes, where no row of ones makes it
    TcUnit<TYPE> unit[tc_halves(TYPE)];  // (only the minimums are used)
    uint32_t info;                       // the step's activation scales and group sums
    int kh;                              // the half, where a unit has one
};

// The sums of a row over the activation rows, in pairs for packed arithmetic (one activation row: the pair's upper half idles).
template <int MC>
struct TcAcc {
    f32x2 v[(MC + 1) / 2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < (MC + 1) / 2; ++i) v[i] = 0ull;
    }
    __device__ __forceinline__ void get(float (&f)[MC]) const {
#pragma unroll
        for (int i = 0; i < (MC + 1) / 2; ++i) {
            float lo, hi;
            unpack2(v[i], lo, hi);
            f[2 * i] = lo;
            if (2 * i + 1 < MC) f[2 * i + 1] = hi;
        }
    }
};

// Sums over the six planes of bytes, of the K activation rows from t0 on, at tensor-memory column d_at.  (MC = 1: beside them the sum of A
// where a row of ones makes it, for there is room for it in the load.)
template <int MC, int K>
__device__ __forceinline__ void tc_load_planes(uint32_t d_at, int t0, uint32_t (&v)[kTcPlanes][K], uint32_t &ones) {
    if constexpr (MC == 1) {
        uint32_t w[8];
        tc::ld8(d_at, w);
#pragma unroll
        for (int i = 0; i < kTcPlanes; ++i) v[i][0] = w[i];
        ones = w[kTcPlanes];
    } else if constexpr (MC == 2) {
        uint32_t w[16];
        tc::ld8(d_at, w);
        tc::ld8(d_at + 8, w + 8);
#pragma unroll
        for (int i = 0; i < 2 * kTcPlanes; ++i) v[i >> 1][i & 1] = w[i];
        ones = w[2 * kTcPlanes];
    } else {
        static_assert(K == 4, "four activation rows");
#pragma unroll
        for (int i = 0; i < kTcPlanes; ++i) tc::ld4(d_at + i * MC + t0, v[i]);
    }
}
// The sum over a piece (exact) and 2^-15 of the sum over the next.
__device__ __forceinline__ float tc_join(uint32_t sum, uint32_t next) {
    return fmaf(static_cast<float>(static_cast<int>(next)), 0x1p-15f, static_cast<float>(static_cast<int>(sum)));
}

// The sums of scaled bytes: with D_p the sums over plane p and S the sum of A,
//   sum of weight * p_q = 2^8 D_2q + D_2q+1 - 2^15 S - offset * sum of p_q,
// exact in 32 bits (modulo 2^32 on the way): |weight| <= 128 or 0 <= weight <= 180, |p_q| <= 2^14, 256 columns.
template <int TYPE, int MC>
__device__ __forceinline__ void tc_accumulate_bytes(const TcPending<TYPE, MC> &p, uint32_t d_at, TcAcc<MC> &acc) {
    static_assert(tc_sums<TYPE, MC>() == 1, "one sum per unit");
    constexpr int kStep = MC > 4 ? 4 : MC, kMins = tc_mins(TYPE);  // activation rows at a time, for the registers' sake
    uint32_t ones = p.ones;
    if constexpr (tc_ones_row(TYPE, MC) && MC > 2) tc::ld1(d_at + kTcPlanes * MC, ones);
#pragma unroll
    for (int t0 = 0; t0 < MC; t0 += kStep) {
        uint32_t v[kTcPlanes][kStep], c[4][kStep];  // c: factors, -offset * sums of the pieces
        tc_load_planes<MC, kStep>(d_at, t0, v, ones);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i > 0 && tc_byte_offset(TYPE) == 0) {
#pragma unroll
                for (int t = 0; t < kStep; ++t) c[i][t] = 0u;
            } else if constexpr (MC == 1) {
                c[i][0] = lds32(p.info + i * tc_info_rows(MC) * 4);
            } else if constexpr (MC == 2) {
                const unsigned long long w = lds64(p.info + i * tc_info_rows(MC) * 4);
                c[i][0] = static_cast<uint32_t>(w), c[i][1] = static_cast<uint32_t>(w >> 32);
            } else {
                const uint4 w = lds128u(p.info + (i * tc_info_rows(MC) + t0) * 4);
                c[i][0] = w.x, c[i][1] = w.y, c[i][2] = w.z, c[i][3] = w.w;
            }
        }
        tc::wait_ld();
        auto value = [&](int t) {
            uint32_t s[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) s[q] = v[2 * q][t] * 256u + v[2 * q + 1][t] + (c[1 + q][t] - 32768u * ones);
            return fmaf(tc_join(s[1], s[2]), 0x1p-15f, static_cast<float>(static_cast<int>(s[0])));
        };
        if constexpr (MC == 1) {
            float a, b;
            unpack2(acc.v[0], a, b);
            acc.v[0] = pack2(fmaf(value(0) * p.s[0], __uint_as_float(c[0][0]), a), b);
        } else {
            const f32x2 s2 = pack2(p.s[0], p.s[0]);
#pragma unroll
            for (int t = 0; t < kStep; t += 2)
                acc.v[(t0 + t) / 2] = fma2(mul2(pack2(value(t), value(t + 1)), s2), pack2(__uint_as_float(c[0][t]), __uint_as_float(c[0][t + 1])), acc.v[(t0 + t) / 2]);
        }
    }
    if constexpr (kMins > 0) {
        auto one = [&](auto tag) {
            constexpr int G = decltype(tag)::value;
            if constexpr (G < kMins) {
                const float m = -p.unit[0].template minimum<G>();
                const uint32_t at = p.info + (tc_info_scales(TYPE, MC) + G * MC) * 4;
                if constexpr (MC == 1) {
                    float a, b;
                    unpack2(acc.v[0], a, b);
                    acc.v[0] = pack2(fmaf(m, __uint_as_float(lds32(at)), a), b);
                } else if constexpr (MC == 2) {
                    acc.v[0] = fma2(pack2(m, m), lds64(at), acc.v[0]);
                } else {
#pragma unroll
                    for (int t = 0; t < MC; t += 4) {
                        const ulonglong2 w = lds128(at + t * 4);
                        acc.v[t / 2] = fma2(pack2(m, m), w.x, acc.v[t / 2]);
                        acc.v[t / 2 + 1] = fma2(pack2(m, m), w.y, acc.v[t / 2 + 1]);
                    }
                }
            }
        };
        one(TcInt<0>{}), one(TcInt<1>{}), one(TcInt<2>{}), one(TcInt<3>{}), one(TcInt<4>{}), one(TcInt<5>{}), one(TcInt<6>{}), one(TcInt<7>{});
        one(TcInt<8>{}), one(TcInt<9>{}), one(TcInt<10>{}), one(TcInt<11>{}), one(TcInt<12>{}), one(TcInt<13>{}), one(TcInt<14>{}), one(TcInt<15>{});
    }
}

// acc[t] += scale * (h0 + 2^-11 h1 + 2^-22 h2 sums) * activation scale  -  minimums * group sums
template <int TYPE, int MC>
__device__ __forceinline__ void tc_accumulate_halves(const TcPending<TYPE, MC> &p, uint32_t d_at, TcAcc<MC> &acc) {
    static_assert(tc_sums<TYPE, MC>() == 1, "one sum per unit");
    constexpr int kMins = tc_mins(TYPE);
    if constexpr (MC > 8) {  // eight activation rows at a time, for the registers' sake
        const f32x2 s2 = pack2(p.s[0], p.s[0]), c1 = pack2(0x1p-11f, 0x1p-11f), c2 = pack2(0x1p-22f, 0x1p-22f);
#pragma unroll
        for (int t0 = 0; t0 < MC; t0 += 8) {
            float v0[8], v1[8], v2[8];
            tc::ld8(d_at + t0, v0);
            tc::ld8(d_at + MC + t0, v1);
            tc::ld8(d_at + 2 * MC + t0, v2);
            const ulonglong2 ia = lds128(p.info + t0 * 4), ib = lds128(p.info + t0 * 4 + 16);
            const f32x2 inv[4] = {ia.x, ia.y, ib.x, ib.y};
            tc::wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                f32x2 u = fma2(pack2(v1[2 * i], v1[2 * i + 1]), c1, pack2(v0[2 * i], v0[2 * i + 1]));
                u = fma2(pack2(v2[2 * i], v2[2 * i + 1]), c2, u);
                acc.v[t0 / 2 + i] = fma2(mul2(u, s2), inv[i], acc.v[t0 / 2 + i]);
            }
        }
        if constexpr (kMins > 0) {
#pragma unroll
            for (int h = 0; h < tc_halves(TYPE); ++h) {
                auto one = [&](auto tag) {
                    constexpr int G = decltype(tag)::value;
                    if constexpr (G < kMins) {
                        const float m = -p.unit[h].template minimum<G>();
                        const uint32_t at = p.info + (tc_info_scales(TYPE, MC) + ((tc_wide(TYPE) ? h : p.kh) * kMins + G) * MC) * 4;
#pragma unroll
                        for (int t = 0; t < MC; t += 4) {
                            const ulonglong2 w = lds128(at + t * 4);
                            acc.v[t / 2] = fma2(pack2(m, m), w.x, acc.v[t / 2]);
                            acc.v[t / 2 + 1] = fma2(pack2(m, m), w.y, acc.v[t / 2 + 1]);
                        }
                    }
                };
                one(TcInt<0>{}), one(TcInt<1>{}), one(TcInt<2>{}), one(TcInt<3>{});
                one(TcInt<4>{}), one(TcInt<5>{}), one(TcInt<6>{}), one(TcInt<7>{});
            }
        }
        return;
    }
    float v[3 * MC + 1];
    tc::ld_sums<MC>(d_at, v);
    f32x2 inv[(MC + 1) / 2];
    if constexpr (MC == 1) {
        inv[0] = pack2(__uint_as_float(lds32(p.info)), 0.0f);
    } else if constexpr (MC == 2) {
        inv[0] = lds64(p.info);
    } else {
#pragma unroll
        for (int t = 0; t < MC; t += 4) {
            const ulonglong2 w = lds128(p.info + t * 4);
            inv[t / 2] = w.x, inv[t / 2 + 1] = w.y;
        }
    }
    tc::wait_ld();
    const float s = p.s[0];
    if constexpr (MC == 1) {
        float a, b, k, unused;
        unpack2(acc.v[0], a, b);
        unpack2(inv[0], k, unused);
        a = fmaf(fmaf(v[2], 0x1p-22f, fmaf(v[1], 0x1p-11f, v[0])) * s, k, a);
        acc.v[0] = pack2(a, b);
    } else {
        const f32x2 s2 = pack2(s, s), c1 = pack2(0x1p-11f, 0x1p-11f), c2 = pack2(0x1p-22f, 0x1p-22f);
#pragma unroll
        for (int t = 0; t < MC; t += 2) {
            f32x2 u = fma2(pack2(v[MC + t], v[MC + t + 1]), c1, pack2(v[t], v[t + 1]));
            u = fma2(pack2(v[2 * MC + t], v[2 * MC + t + 1]), c2, u);
            acc.v[t / 2] = fma2(mul2(u, s2), inv[t / 2], acc.v[t / 2]);
        }
    }
    if constexpr (kMins > 0) {
#pragma unroll
        for (int h = 0; h < tc_halves(TYPE); ++h) {
            float sums[kMins * MC];
#pragma unroll
            for (int i = 0; i < kMins * MC; i += 4) {
                const uint4 w = lds128u(p.info + (tc_info_scales(TYPE, MC) + (tc_wide(TYPE) ? h : p.kh) * kMins * MC + i) * 4);
                sums[i] = __uint_as_float(w.x), sums[i + 1] = __uint_as_float(w.y), sums[i + 2] = __uint_as_float(w.z), sums[i + 3] = __uint_as_float(w.w);
            }
            auto one = [&](auto tag) {
                constexpr int G = decltype(tag)::value;
                if constexpr (G < kMins) {
                    const float m = -p.unit[h].template minimum<G>();
                    if constexpr (MC == 1) {
                        float a, b;
                        unpack2(acc.v[0], a, b);
                        acc.v[0] = pack2(fmaf(m, sums[G], a), b);
                    } else {
#pragma unroll
                        for (int t = 0; t < MC; t += 2) acc.v[t / 2] = fma2(pack2(m, m), pack2(sums[G * MC + t], sums[G * MC + t + 1]), acc.v[t / 2]);
                    }
                }
            };
            one(TcInt<0>{}), one(TcInt<1>{}), one(TcInt<2>{}), one(TcInt<3>{});
            one(TcInt<4>{}), one(TcInt<5>{}), one(TcInt<6>{}), one(TcInt<7>{});
        }
    }
}

// Sums of a unit over its groups of 32 columns, for types with integer scales: scale * sum of weight * p0, exactly (127 * 2^11 * 32 columns
// times 32, times 8 groups: below 2^31), and of the rest.
template <int TYPE, int MC>
struct TcUnitSums {
    int top[tc_integer_scale(TYPE) ? MC : 1];
    float rest[tc_integer_scale(TYPE) ? MC : 1];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int &x : top) x = 0;
#pragma unroll
        for (float &x : rest) x = 0.0f;
    }
};
// The sums of signed bytes, one per 32 columns: with D_p the sums over plane p, sum of weight * p_q = 2^8 D_2q + D_2q+1, at most 2^26.
//   last: these are a unit's last sums
template <int TYPE, int MC>
__device__ __forceinline__ void tc_accumulate_blocks(const TcPending<TYPE, MC> &p, uint32_t d_at, bool last, TcUnitSums<TYPE, MC> &unit, TcAcc<MC> &acc) {
    constexpr int kSums = tc_sums<TYPE, MC>(), kN = TcShape<TYPE, MC>::kN;
    constexpr int kStep = MC > 4 ? 4 : MC, kAtOnce = MC == 1 ? kSums : MC == 2 && !tc_integer_scale(TYPE) ? 2 : 1;  // rows and sums at a time (registers)
#pragma unroll
    for (int t0 = 0; t0 < MC; t0 += kStep) {
        f32x2 inv[(kStep + 1) / 2];
        if (!tc_integer_scale(TYPE) || last) {
            if constexpr (MC == 1) {
                inv[0] = pack2(__uint_as_float(lds32(p.info)), 0.0f);
            } else if constexpr (MC == 2) {
                inv[0] = lds64(p.info);
            } else {
                const ulonglong2 w = lds128(p.info + t0 * 4);
                inv[0] = w.x, inv[1] = w.y;
            }
        }
        auto add = [&](float s, const float (&u)[kStep]) {
            if constexpr (MC == 1) {
                float a, b, k, none;
                unpack2(acc.v[0], a, b);
                unpack2(inv[0], k, none);
                acc.v[0] = pack2(fmaf(u[0] * s, k, a), b);
            } else {
#pragma unroll
                for (int t = 0; t < kStep; t += 2)
                    acc.v[(t0 + t) / 2] = fma2(mul2(pack2(u[t], u[t + 1]), pack2(s, s)), inv[t / 2], acc.v[(t0 + t) / 2]);
            }
        };
#pragma unroll
        for (int g0 = 0; g0 < kSums; g0 += kAtOnce) {
            uint32_t v[kAtOnce][kTcPlanes][kStep], unused;
#pragma unroll
            for (int g = 0; g < kAtOnce; ++g) tc_load_planes<MC, kStep>(d_at + (g0 + g) * kN, t0, v[g], unused);
            tc::wait_ld();
#pragma unroll
            for (int g = 0; g < kAtOnce; ++g) {
                float u[kStep];
#pragma unroll
                for (int t = 0; t < kStep; ++t) {
                    const uint32_t p0 = v[g][0][t] * 256u + v[g][1][t], p1 = v[g][2][t] * 256u + v[g][3][t], p2 = v[g][4][t] * 256u + v[g][5][t];
                    if constexpr (tc_integer_scale(TYPE)) {
                        const int k = __float_as_int(p.s[g0 + g]);
                        unit.top[t0 + t] += k * static_cast<int>(p0);
                        unit.rest[t0 + t] = fmaf(tc_join(p1, p2), static_cast<float>(k), unit.rest[t0 + t]);
                    } else {
                        u[t] = fmaf(tc_join(p1, p2), 0x1p-15f, static_cast<float>(static_cast<int>(p0)));
                    }
                }
                if constexpr (!tc_integer_scale(TYPE)) add(p.s[g0 + g], u);
            }
        }
        if constexpr (tc_integer_scale(TYPE)) {
            if (last) {
                float u[kStep];
#pragma unroll
                for (int t = 0; t < kStep; ++t) {
                    u[t] = fmaf(unit.rest[t0 + t], 0x1p-15f, static_cast<float>(unit.top[t0 + t]));
                    unit.rest[t0 + t] = 0.0f, unit.top[t0 + t] = 0;
                }
                add(p.d, u);
            }
        }
    }
}

template <int TYPE, int MC>
__device__ __forceinline__ void tc_accumulate(const TcPending<TYPE, MC> &p, uint32_t d_at, bool last, TcUnitSums<TYPE, MC> &unit, TcAcc<MC> &acc) {
    if constexpr (tc_scaled_bytes(TYPE)) tc_accumulate_bytes<TYPE, MC>(p, d_at, acc);
    else if constexpr (tc_bytes(TYPE)) tc_accumulate_blocks<TYPE, MC>(p, d_at, last, unit, acc);
    else tc_accumulate_halves<TYPE, MC>(p, d_at, acc);
}

// One output weight by weight, for sums that came out as no number: an infinite or undefined activation has no exact planes, and
// a weight in two parts, or with a minimum beside it, turns an infinity into the difference of two.  What is returned is
// infinite or undefined where the weights and the activations themselves make it so.  One thread per output, uncoalesced: an LM
// head of 151936 x 5120 whose 8 rows are all undefined takes 17 ms instead of 0.2; the check alone costs up to 0.6 % (a layer of
// 4 rows with prologues 88.7 -> 89.2 us).
template <int TYPE>
__device__ __noinline__ float tc_plain_sum(const MatvecArgs &a, const uint8_t *row, int t, float factor) {
    constexpr int kChunks = chunk_block(TYPE) / 8;
    const uint8_t *table = grid_is_codebook(TYPE) ? a.codebook : reinterpret_cast<const uint8_t *>(kIq4Levels);
    const size_t x0 = static_cast<size_t>(t) * a.cols;
    float sum = 0.0f;
#pragma unroll 1
    for (int c = 0; c < a.cols / 8; ++c) {
        float w[8];
        deq8<TYPE>(row + static_cast<size_t>(c / kChunks) * chunk_block_bytes(TYPE), c % kChunks, w, table);
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
            const int col = 8 * c + i;
            float x = a.x[x0 + col];
            if (a.fuse & kFuseSiluMul) x = x / (1.0f + expf(-x)) * a.x2[x0 + col];
            if (a.fuse & kFuseNorm) x *= factor * a.norm_w[col];
            sum = fmaf(w[i], x, sum);
        }
    }
    return sum;
}

__device__ __forceinline__ bool tc_better(float v, int i, float bv, int bi) { return v > bv || (v == bv && i < bi); }

// The order of floats as unsigned integers (no NaN).
__device__ __forceinline__ uint32_t tc_ordered(float v) {
    const uint32_t b = __float_as_uint(v);
    return b ^ ((static_cast<uint32_t>(static_cast<int32_t>(b) >> 31)) | 0x80000000u);
}
// Fused argmax: what a warp's lanes have put out for an activation row (rows ascend with the lanes) against the warp's best so far.
// NaN is no output; ties to the lower row.
__device__ __forceinline__ void tc_note_best(bool exists, float v, int row, int lane, float *best_v, int *best_i) {
    const uint32_t key = exists && v == v ? tc_ordered(v == 0.0f ? 0.0f : v) : 0u;
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, key);
    const uint32_t who = __ballot_sync(0xFFFFFFFFu, key == top);
    if (top != 0u && lane == __ffs(static_cast<int>(who)) - 1 && tc_better(v, row, *best_v, *best_i)) *best_v = v, *best_i = row;
    __syncwarp();
}

// Block partials, then the last block to finish reduces them (ties to the lowest row, 0x7fffffff if nothing is above -inf).
__device__ __forceinline__ void tc_finish_argmax(const TcMatvecArgs &a, int m, int warp, int lane, const float (*s_v)[8], const int (*s_i)[8], bool *s_last) {
    __syncthreads();
    const int grid = static_cast<int>(gridDim.x);
    if (threadIdx.x < static_cast<unsigned>(m)) {
        const int t = static_cast<int>(threadIdx.x);
        float bv = s_v[0][t];
        int bi = s_i[0][t];
        for (int w = 1; w < 16; ++w)
            if (tc_better(s_v[w][t], s_i[w][t], bv, bi)) bv = s_v[w][t], bi = s_i[w][t];
        a.part_val[t * grid + blockIdx.x] = bv;
        a.part_idx[t * grid + blockIdx.x] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        *s_last = atomicAdd(a.done_counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    if (warp < m) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int b = lane; b < grid; b += 32) {
            const float v = __ldcg(a.part_val + warp * grid + b);
            const int i = __ldcg(a.part_idx + warp * grid + b);
            if (tc_better(v, i, bv, bi)) bv = v, bi = i;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, off);
            const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
            if (tc_better(ov, oi, bv, bi)) bv = ov, bi = oi;
        }
        if (lane == 0) {
            bi = bi == 0x7fffffff ? bi : bi + a.row_base;
            // a launch that takes the last tiles of a tensor: the launch before it has left the best of the others, all lower rows
            if (a.tc_first == 0 || bv > a.out_val[warp]) {
                a.out_idx[warp] = bi;
                if (a.out_val != nullptr) a.out_val[warp] = bv;
            }
        }
    }
    if (threadIdx.x == 0) *a.done_counter = 0;
}

// An output: the sum over all columns, its epilogue, the store.
template <int TYPE>
__device__ __forceinline__ float tc_put(const TcMatvecArgs &a, const MatvecPart &part, int row, int t, float sum, float factor) {
    if (a.fuse & kFuseNorm) sum *= factor;
    if (sum != sum) sum = tc_plain_sum<TYPE>(a, part.w + static_cast<size_t>(row) * a.row_bytes, t, factor);
    if (part.y != nullptr) {
        float *y = part.y + static_cast<size_t>(t) * part.rows + row;
        if (a.fuse & kFuseAdd) sum += *y;
        *y = sum;
    }
    return sum;
}

// A word of a.partials that nobody has written: a NaN that no arithmetic gives.
constexpr uint32_t kTcEmpty = 0xFFFFFFFFu;
template <int N>
__device__ __forceinline__ void tc_store_words(float *to, const uint32_t (&v)[N]) {
    if constexpr (N == 1) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(to), "r"(v[0]) : "memory");
    else if constexpr (N == 2) asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(to), "r"(v[0]), "r"(v[1]) : "memory");
    else asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(to), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
template <int N>
__device__ __forceinline__ void tc_load_words(const float *from, uint32_t (&v)[N]) {
    if constexpr (N == 1) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v[0]) : "l"(from) : "memory");
    else if constexpr (N == 2) asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(from) : "memory");
    else asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(from) : "memory");
}
__device__ __forceinline__ uint32_t tc_word(float v) {
    const uint32_t b = __float_as_uint(v);
    return b == kTcEmpty ? 0x7FFFFFFFu : b;
}

// Where the sums of row r, activation row t of the exchange (of kOut) and a pair of groups lie in shared memory: a warp stores every eighth
// row and reads 32 rows in turn, both without bank conflicts.
template <int kOut>
__device__ __forceinline__ uint32_t tc_red_at(uint32_t red, int pair, int t, int r) {
    return red + ((pair * kOut + t) * kTcRedRows + r + (r >> 3)) * 4;
}

// Finishes a tile outside of a cluster: all decoder warps, thread = row, the two halves of the threads share the activation rows.
// With columns split, the last of the k_split blocks to have counted itself in (each does so before its last sums are there) adds the
// parts up in the order of the columns; the others leave theirs in a.partials.  They come with no fence: the last block reads words
// until none is empty, and leaves them empty again.  It only waits for blocks that are about to store: blocks may run at any time and in any
// place, and no cluster has to find room at once (120 blocks in clusters of 6 leave 28 SMs, of which other clusters cannot use most).
// The way through L2 takes some 0.5 us longer than one through a cluster's shared memory, which a stream alone notices (back to back, a layer of
// 4 rows 94.2 -> 98.6 us, one of 8 106.9 -> 114.2), so it has clusters; three streams that share the GPU do not: clusters and this, each with
// launch_dependents where it is now, layers of 1, 4 (fused) and 8 rows 67.3 / 81.9 / 81.2 and 60.8 / 73.3 / 75.0 us, 24 rows of three tensors
// 101 and 84, six tensors of odd sizes with 2 rows 62 and 53.
// (What was slower: a warp at a time, each with its own count, M=8 Q6_K 1024 x 5120 10.6 -> 11.8 us; counts that acquire and release, or fences on both
// sides of a relaxed one, 0.6 and 1.4 us more.)
// The loop over the outputs is rolled: this code runs once per tile, its instructions come from L2.
template <int TYPE, int MC>
__device__ __forceinline__ void tc_finish_tile(const TcMatvecArgs &a, int m, int p, int tile, int tile_row, int rank, bool more, uint32_t red, const float (&sums)[MC],
                                               const float *norm, const int *s_last, float (*best_v)[8], int (*best_i)[8], volatile int *failed) {
    constexpr int kOut = tc_out_rows(MC), kHalf = (kOut + 1) / 2, kVec = kHalf < 4 ? kHalf : 4;  // activation rows per exchange, a thread's part of them
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = threadIdx.x & 255, half = threadIdx.x >> 8, k_split = a.k_split;
    const MatvecPart &part = a.part[p];
    const int row = tile_row * kTcRows + r;
    const bool exists = row < part.rows;
    unsigned long long began = 0;
#pragma unroll
    for (int round = 0; round < MC / kOut; ++round) {
        {
            const int mine = ((warp >> 2) & 1) * 4 + (warp & 3) + 8 * lane;
#pragma unroll
            for (int t = 0; t < kOut; ++t)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(tc_red_at<kOut>(red, warp >> 3, t, mine)), "f"(sums[round * kOut + t]) : "memory");
        }
        tc::decoders_sync();
        const int t0 = round * kOut + half * kHalf;  // the thread's activation rows: kHalf from here on
        if (t0 < m && (MC > 1 || half == 0)) {
            const uint32_t at = tc_red_at<kOut>(red, 0, half * kHalf, r);
            constexpr uint32_t kNext = kTcRedRows * 4, kPair = kOut * kNext;
            float sq = 0.0f;  // lane i: the squares of activation row t0 + i
            if (a.fuse & kFuseNorm) sq = lane < kHalf ? norm[t0 + lane] : 0.0f;
            if (a.fuse & kFuseAdd) {  // what the outputs are added to, so that they do not wait for one row after the other
#pragma unroll 1
                for (int t = t0; t < t0 + kHalf && t < m; ++t)
                    if (exists) asm volatile("prefetch.global.L1 [%0];" ::"l"(part.y + static_cast<size_t>(t) * part.rows + row));
            }
            bool out = true;
            if (k_split > 1) {
                // [round][column range][half]: [256 rows][kHalf], then for each of 8 warps the squares
                constexpr int kRecord = kHalf * kTcRows + 32;
                float *const first = a.partials + (((tile - a.tc_first) * (MC / kOut) + round) * k_split * 2 + half) * kRecord;
                out = *s_last == k_split - 1;
                uint32_t own[kHalf];
#pragma unroll
                for (int i = 0; i < kHalf; ++i) own[i] = tc_word(__uint_as_float(lds32(at + i * kNext)) + __uint_as_float(lds32(at + i * kNext + kPair)));
                if (!out) {
                    tc_store_words(first + rank * 2 * kRecord + r * kHalf, own);
                    if ((a.fuse & kFuseNorm) && lane < kHalf) {
                        const uint32_t w[1] = {tc_word(sq)};
                        tc_store_words(first + rank * 2 * kRecord + kHalf * kTcRows + (warp & 7) * 4 + lane, w);
                    }
                } else {
                    // the squares, lane 4 k + i: of column range k
                    float *const squares = first + (lane >> 2) * 2 * kRecord + kHalf * kTcRows + (warp & 7) * 4 + (lane & 3);
                    const bool there = (a.fuse & kFuseNorm) && lane < 4 * k_split && (lane & 3) < kHalf && (lane >> 2) != rank;
                    uint32_t w[1] = {0u};
                    uint32_t v[kMaxSplit][kVec];
                    static_assert(kHalf == kVec, "one load per column range");
                    float *const from = first + r * kHalf;
#pragma unroll 1
                    for (uint32_t i = 1;; ++i) {
                        if (there) tc_load_words(squares, w);
#pragma unroll
                        for (int k = 0; k < kMaxSplit; ++k) {
#pragma unroll
                            for (int j = 0; j < kVec; ++j) v[k][j] = 0u;
                            if (k < k_split && k != rank) tc_load_words(from + k * 2 * kRecord, v[k]);
                        }
                        bool empty = w[0] == kTcEmpty;
#pragma unroll
                        for (int k = 0; k < kMaxSplit; ++k)
#pragma unroll
                            for (int j = 0; j < kVec; ++j) empty |= v[k][j] == kTcEmpty;
                        if (!__any_sync(0xFFFFFFFFu, empty) || ((i & 255u) == 0 && __any_sync(0xFFFFFFFFu, tc::give_up(&began, failed)))) break;
                    }
#pragma unroll
                    for (int j = 0; j < kVec; ++j) {
                        float sum = 0.0f;
#pragma unroll
                        for (int k = 0; k < kMaxSplit; ++k) sum += __uint_as_float(k == rank ? own[j] : v[k][j]);
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + j * kNext), "f"(sum) : "memory");
                    }
                    if (a.fuse & kFuseNorm) {
                        const uint32_t none[1] = {kTcEmpty};
                        if (there) tc_store_words(squares, none);
                        const float mine = __shfl_sync(0xFFFFFFFFu, sq, lane & 3);
                        if ((lane >> 2) == rank) w[0] = __float_as_uint(mine);
                        sq = 0.0f;
#pragma unroll 1
                        for (int k = 0; k < k_split; ++k) sq += __uint_as_float(__shfl_sync(0xFFFFFFFFu, w[0], 4 * k + (lane & 3)));
                    }
                    uint32_t none[kVec];
#pragma unroll
                    for (int j = 0; j < kVec; ++j) none[j] = kTcEmpty;
#pragma unroll 1
                    for (int k = 0; k < k_split; ++k) {
                        if (k != rank) tc_store_words(from + k * 2 * kRecord, none);
                    }
                }
            }
            if (out) {
                const float scale = (a.fuse & kFuseNorm) ? 1.0f / sqrtf(sq / static_cast<float>(a.cols) + a.eps) : 1.0f;
                uint32_t from = at;
#pragma unroll 1
                for (int i = 0; i < kHalf && t0 + i < m; ++i, from += kNext) {
                    float sum = __uint_as_float(lds32(from));
                    if (k_split == 1) sum += __uint_as_float(lds32(from + kPair));
                    const float factor = __shfl_sync(0xFFFFFFFFu, scale, i);
                    if (exists) sum = tc_put<TYPE>(a, part, row, t0 + i, sum, factor);
                    if (a.out_idx != nullptr) tc_note_best(exists, sum, row, lane, &best_v[warp][t0 + i], &best_i[warp][t0 + i]);
                }
            }
        }
        if (more || round + 1 < MC / kOut) tc::decoders_sync();  // the sums may be overwritten
    }
}

// B operands and infos of the activation rows t0 .. t0 + 15 below m, of MC, one block per step: what every block of the matvec would work
// out for itself.
template <int TYPE, int MC>
__global__ void __launch_bounds__(16 * 32) tc_split_kernel(const __grid_constant__ MatvecArgs a, uint8_t *out, const int t0, const int m) {
    constexpr int kOperand = TcShape<TYPE, MC>::kGroupsB * tc_group_b(TYPE), kBytes = tc_split_bytes<TYPE, MC>();
    __shared__ __align__(16) uint8_t image[kBytes];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int step = blockIdx.x, t = t0 + static_cast<int>(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
    if (t < m) {
        TcColumns c;
        tc_fetch<TYPE>(a, t, step * kTcStepCols, cols_here, lane, c);
        tc_convert<TYPE, MC, true>(a, c, t, step * kTcStepCols, cols_here, tc::s32(image), tc::s32(image) + kOperand, 0u, lane);
    }
    __syncthreads();
    uint4 *to = reinterpret_cast<uint4 *>(out + static_cast<size_t>(step) * kBytes);
    for (int i = threadIdx.x; i < kBytes / 16; i += 16 * 32) {
        if constexpr (MC > 16) {  // a launch's share: whole groups of 8 B rows, and 4 of every MC floats at a time
            const int row = i < kOperand / 16 ? i / (tc_group_b(TYPE) / 16) * 8 % MC : (i - kOperand / 16) * 4 % MC;
            if (row < t0 || row >= t0 + 16) continue;
        }
        to[i] = reinterpret_cast<const uint4 *>(image)[i];
    }
}

template <int TYPE, int MC, typename MAPS>
__global__ void __launch_bounds__(kTcThreads, 1) tcmv_kernel(const __grid_constant__ TcMatvecArgs a, const __grid_constant__ MAPS maps, const int m) {
    using Shape = TcShape<TYPE, MC>;
    constexpr int kStages = tc_stages<TYPE, MC>(), kStageBytes = tc_stage_bytes<TYPE, MC>();
    constexpr int kPitch = tc_pitch(TYPE), kStepBytes = tc_step_bytes(TYPE);
    constexpr int kNB = tc_b_stages<TYPE, MC>();
    constexpr bool kWide = tc_wide(TYPE), kPresplit = tc_presplit(MC);
    constexpr int kOut = tc_out_rows(MC);  // activation rows whose sums go out together
    constexpr uint32_t kTmD = tc_chunk_regs(TYPE) * tc_batch_chunks<TYPE, MC>();  // a group's sums start at this column of its 128
    constexpr uint32_t kIdesc = tc::instruction(TYPE, Shape::kN);
    static_assert(kTmD + tc_sums<TYPE, MC>() * Shape::kN <= 128, "tensor memory of a group");
    static_assert(kStages >= (kWide ? 3 : 2) && kStages + 2 <= kTcInfoSlots, "stage ring");
    extern __shared__ uint8_t tc_raw[];
    __shared__ __align__(8) uint64_t s_wfull[6], s_wempty[6], s_bfull[4], s_bempty[4], s_afull[4], s_done[4], s_cluster, s_read;
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ float s_norm[kMaxSplit][8];  // sums of squares of the activation rows, from every block of the cluster
    __shared__ float s_best_v[16][8];  // fused argmax: the best outputs that each warp has seen, per activation row
    __shared__ int s_best_i[16][8];
    __shared__ bool s_last;
    __shared__ int s_count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // layout: stages (1024-byte aligned) | table | B ring | per-step info | sums of the tile | sums of squares
    const uint32_t stages = (tc::s32(tc_raw) + 1023u) & ~1023u;
    [[maybe_unused]] const uint32_t table = stages + kStages * kStageBytes;
    const uint32_t b_ring = table + (tc_table_bytes(TYPE, MC) + 127) / 128 * 128;
    const uint32_t info_ring = b_ring + (kNB * Shape::kGroupsB + 1) * tc_group_b(TYPE);
    const uint32_t red = info_ring + kTcInfoSlots * tc_info_floats(TYPE, MC) * 4;
    const uint32_t norm_parts = red + 2 * kTcRedRows * kOut * 4;
    volatile int *failed = &s_failed;

    const int k_split = a.k_split;
    const bool clustered = k_split > 1 && a.partials == nullptr;
    int group = static_cast<int>((blockIdx.x * static_cast<unsigned>(a.tc_split_recip)) >> 16), n_groups = a.tc_groups;
    const int rank = static_cast<int>(blockIdx.x) - group * k_split;
    const int step0 = a.tc_steps[rank], step1 = a.tc_steps[rank + 1];
    constexpr bool kSingle = sizeof(MAPS) == sizeof(TcMaps1);  // one tensor: nothing to look up
    auto tiles_of = [&](int p) { return (a.part[p].rows + kTcRows - 1) / kTcRows; };
    const int end0 = kSingle ? 0 : tiles_of(0), end1 = kSingle ? 0 : end0 + tiles_of(1), end2 = kSingle ? 0 : end1 + tiles_of(2), n_tiles = a.tc_end;
    group += a.tc_first;
    // the tensor a tile belongs to, and that tensor's first tile
    auto part_of = [&](int tile) { return kSingle ? 0 : (tile >= end0) + (tile >= end1) + (tile >= end2); };
    auto first_tile = [&](int p) { return kSingle || p == 0 ? 0 : p == 1 ? end0 : p == 2 ? end1 : end2; };

    // ---- copy side: stage s of a step holds, per row class, 32 rows of kPitch bytes, then the activation rows ----
    auto class_mis = [&](const MatvecPart &p, int c) {
        return static_cast<uint32_t>((reinterpret_cast<uintptr_t>(p.w) + static_cast<uintptr_t>(c) * static_cast<uintptr_t>(a.row_bytes)) & 15u);
    };
    // Weights pass through L2 once; they should not take the place of activations, sums and code.  (16 layers in one graph, 4 and 8 rows: 74.2 and
    // 89.1 us a layer, 72.6 and 85.6 so; passes on three streams 0 to 3 % faster.)
    uint64_t once;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    auto copy_weights = [&](int tile, int step, int stage, bool with_x) {  // one thread
        const int p = part_of(tile), y = (tile - first_tile(p)) * 32;
        const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
        const uint32_t bar = tc::s32(&s_wfull[stage]), at = stages + stage * kStageBytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kTcRows * kPitch + (with_x && !kPresplit ? m * cols_here * 4 : 0))
                     : "memory");
        const int shift = a.tc_map_shift[p];  // map c of n brings classes c, c + n, c + 2n, ...
#pragma unroll 1
        for (int c = 0; c < 1 << shift; ++c) {
            const uint32_t x = ((class_mis(a.part[p], c) + static_cast<uint32_t>(step) * kStepBytes) & ~15u) / kTcElemBytes;
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(
                             at + ((c * 8) >> shift) * 32 * kPitch),
                         "l"(&maps.m[p][c]), "r"(x), "r"(y), "r"(0), "r"(bar), "l"(once)
                         : "memory");
        }
    };
    auto copy_x = [&](int step, int stage) {  // one thread
        const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
        if constexpr (kPresplit) return;
        for (int t = 0; t < m; ++t)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             stages + stage * kStageBytes + kTcRows * kPitch + t * (kTcStepCols * 4)),
                         "l"(a.x + static_cast<size_t>(t) * a.cols + step * kTcStepCols), "r"(cols_here * 4), "r"(tc::s32(&s_wfull[stage]))
                         : "memory");
    };

    // Set-up: the copy warp requests the first stages and does not wait for anybody; the other warps meanwhile load the first steps'
    // activations.  (A block's first MMAs came 7800 cycles after its start, of which weights take 4700: everybody waited 1300 cycles for
    // the requests to be issued, and activations requested behind 150 KB of weights came 2500 cycles later.  Now 5400.  17408 x 5120,
    // 1 row: Q3_K 15.7 -> 15.3 us, Q4_K 15.7 -> 15.0.)
    constexpr int kFirst = kPresplit ? 0 : (kNB * MC + 15) / 16;  // conversions of a warp before the loop
    [[maybe_unused]] TcColumns first[kFirst == 0 ? 1 : kFirst];
    int copy_tile = group, copy_step = step0, copied = 0;  // copy warp: the next stage's tile and step
    auto copy_next = [&](int n) {                          // weights never depend on an earlier kernel
#pragma unroll 1
        for (; copied < n && copy_tile < n_tiles; ++copied) {
            copy_weights(copy_tile, copy_step, copied, copied >= kNB);
            if (++copy_step == step1) copy_step = step0, copy_tile += n_groups;
        }
    };
    if (warp == 16) {
        if (tc::elect_one()) {
            for (int s = 0; s < kStages; ++s) tc::bar_init(tc::s32(&s_wfull[s]), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            copy_next(kWide ? 2 : 1);
            for (int s = 0; s < kStages; ++s) tc::bar_init(tc::s32(&s_wempty[s]), kWide ? 8 : 16);
            for (int s = 0; s < kNB; ++s) {
                tc::bar_init(tc::s32(&s_bfull[s]), kPresplit ? 1u : static_cast<uint32_t>(m));
                tc::bar_init(tc::s32(&s_bempty[s]), kWide ? 2 : 4);
            }
            for (int g = 0; g < 4; ++g) {
                tc::bar_init(tc::s32(&s_afull[g]), 4);
                tc::bar_init(tc::s32(&s_done[g]), 1);
            }
            tc::bar_init(tc::s32(&s_cluster), 1);
            tc::bar_init(tc::s32(&s_read), static_cast<uint32_t>(k_split));
            s_failed = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        asm volatile("bar.arrive 6, %0;" ::"n"(kTcThreads) : "memory");
    } else {
        if (warp == 17) {  // the first tile's maps
            const int p = part_of(group);
            if (lane < 1 << a.tc_map_shift[p]) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.m[p][lane]) : "memory");
        } else if (warp == 18) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::s32(&s_tmem)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
            tc::fence_before();
        } else {
            if constexpr (tc_signed_table(TYPE)) {
                tc_make_signed_table<TYPE, MC>(a.codebook, table);
            } else if constexpr (grid_is_codebook(TYPE)) {
                for (int i = threadIdx.x; i < grid_bytes(TYPE) / 16; i += kTcDecoders) {
                    const uint4 w = *reinterpret_cast<const uint4 *>(a.codebook + i * 16);
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(table + i * 16), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
                }
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");  // activations are read and outputs written from here on
#pragma unroll
            for (int i = 0; i < kFirst; ++i) {
                const int n = (warp + 16 * i) / MC, t = (warp + 16 * i) % MC;
                if (n < kNB && t < m) {
                    int step = step0 + n;
                    while (step >= step1) step -= step1 - step0;
                    const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
                    tc_fetch<TYPE>(a, t, step * kTcStepCols, cols_here, lane, first[i]);
                }
            }
        }
        asm volatile("bar.sync 6, %0;" ::"n"(kTcThreads) : "memory");
    }
    // Announces this block's barriers to the cluster; whoever signals them waits for the announcements first.  (The barriers were
    // published by the fence behind their initialisation; a releasing arrive would wait for the copies in flight, 3 us.)
    if (clustered) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    tc::fence_after();

    if (warp == 16) {
        if (tc::elect_one()) {
            copy_next(kStages);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int filled = 0, stage = 0;
            uint32_t phase = 0;
            [[maybe_unused]] int bs = 0;
            [[maybe_unused]] uint32_t bphase = 0;
            for (int tile = group; tile < n_tiles && !*failed; tile += n_groups)
                for (int step = step0; step < step1; ++step) {
                    if (filled >= kStages) {
                        tc::bar_wait(tc::s32(&s_wempty[stage]), phase ^ 1u, failed);
                        if (*failed) break;
                        copy_weights(tile, step, stage, filled >= kNB);
                    }
                    if (filled >= kNB) copy_x(step, stage);
                    if constexpr (kPresplit) {  // the step's B operand and infos
                        constexpr int kOperand = Shape::kGroupsB * tc_group_b(TYPE), kInfo = tc_info_floats(TYPE, MC) * 4;
                        if (filled >= kNB) {
                            tc::bar_wait(tc::s32(&s_bempty[bs]), bphase ^ 1u, failed);
                            if (*failed) break;
                        }
                        const uint8_t *from = a.x_split + static_cast<size_t>(step) * tc_split_bytes<TYPE, MC>();
                        const uint32_t bar = tc::s32(&s_bfull[bs]);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kOperand + kInfo) : "memory");
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                         b_ring + bs * kOperand),
                                     "l"(from), "r"(kOperand), "r"(bar)
                                     : "memory");
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                         info_ring + (filled & (kTcInfoSlots - 1)) * kInfo),
                                     "l"(from + kOperand), "r"(kInfo), "r"(bar)
                                     : "memory");
                        if (++bs == kNB) bs = 0, bphase ^= 1u;
                    }
                    ++filled;
                    if (++stage == kStages) stage = 0, phase ^= 1u;
                }
            // After a wait gave up: the copies already requested must land before the block may leave.  The next fill would go to
            // `stage` in phase `phase`; stages behind it have been filled in that phase, the others in the one before.
            if (*failed) {
#pragma unroll 1
                for (int s = 0; s < kStages; ++s)
                    for (int i = 0; i < 4096 && !tc::bar_try(tc::s32(&s_wfull[s]), s < stage || filled < kStages ? phase : phase ^ 1u); ++i) __nanosleep(64);
                if constexpr (kPresplit) {
#pragma unroll 1
                    for (int s = 0; s < kNB && s < filled; ++s)
                        for (int i = 0; i < 4096 && !tc::bar_try(tc::s32(&s_bfull[s]), s < bs ? bphase : bphase ^ 1u); ++i) __nanosleep(64);
                }
            }
        }
        __syncwarp();
    } else if (warp > 16) {
        // ---- MMA issue: warp 17 for groups 0 and 1, warp 18 for groups 2 and 3 ----
        constexpr int kBC = tc_batch_chunks<TYPE, MC>(), kBatches = tc_halves(TYPE) * tc_half_batches<TYPE, MC>(), kMmas = tc_chunk_regs(TYPE) / 8 * kBC;
        const int pair = warp - 17;
        const uint32_t tmem = s_tmem;
        int bs = 0, st = 0;
        uint32_t bphase = 0, aphase = 0;
        for (int tile = group; tile < n_tiles; tile += n_groups)
            for (int step = step0; step < step1; ++step) {
                if (!kWide || (st & 1) == pair) {
                    const uint64_t b_unit = tc::b_desc<TYPE>(b_ring + bs * (Shape::kGroupsB * tc_group_b(TYPE)) + (kWide ? 0 : pair * (tc_group_b(TYPE) / 2)));
                    tc::bar_wait(tc::s32(&s_bfull[bs]), bphase, failed);
#pragma unroll
                    for (int b = 0; b < kBatches; ++b) {
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            const int wg = 2 * pair + g;
                            tc::bar_wait(tc::s32(&s_afull[wg]), aphase, failed);
                            tc::fence_after();
                            if (tc::elect_one()) {
                                const uint32_t tm = tmem + wg * 128;
#pragma unroll
                                for (int j = 0; j < kMmas; ++j) {
                                    // the B tile of 16 columns behind the batch's j-th 16 A columns (two A tiles per B tile with two parts)
                                    const int i = tc_parts(TYPE) == 2 ? ((b * kBC + (j >> 2)) * 2 + ((j & 3) >> 1)) : b * kMmas + j;
                                    const int sum = tc_block32(TYPE) ? j : 0;
                                    const bool fresh = tc_block32(TYPE) || (b == 0 && j == 0);
                                    tc::mma<TYPE>(tm + kTmD + sum * Shape::kN, tm + j * 8, b_unit + static_cast<uint64_t>(i * (2 * kTcCore / 16)), kIdesc,
                                            fresh ? 0u : 1u);
                                }
                                tc::commit(tc::s32(&s_done[wg]));
                                if (b == kBatches - 1) tc::commit(tc::s32(&s_bempty[bs]));
                            }
                            __syncwarp();
                        }
                        aphase ^= 1u;
                    }
                }
                ++st;
                if (++bs == kNB) bs = 0, bphase ^= 1u;
            }
        if (warp == 18) {  // once the decoders have read the last sums, beside the outputs
            asm volatile("bar.sync 7, %0;" ::"n"(kTcDecoders + 32) : "memory");
            tc::fence_after();
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        }
    } else {
        const int wg = warp >> 2, quarter = warp & 3, rw = wg & 1, pair = wg >> 1, kh = kWide ? 0 : pair;
        const int cls = rw * 4 + quarter;  // this warp's row class: rows cls, cls + 8, ... of the tile
        const uint32_t tm_mine = s_tmem + wg * 128 + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t a_full = tc::s32(&s_afull[wg]), mma_done = tc::s32(&s_done[wg]);
        int st = 0, stage = 0, bs = 0;  // step count, stage, B stage
        uint32_t wphase = 0, bphase = 0, dphase = 1;  // (dphase: of the batch before the next one)
        bool pending = false;    // a unit's sums have not been read yet
        TcPending<TYPE, MC> pend;
        TcUnitSums<TYPE, MC> unit_sums;
        unit_sums.clear();
        TcAcc<MC> acc;
        acc.clear();
        uint32_t rounds = 0;  // in which sums have been handed over
        if (lane < 8) s_best_v[warp][lane] = -INFINITY, s_best_i[warp][lane] = 0x7fffffff;

        // The first kNB steps' activations are converted by all warps at once, straight from global memory: the way through the
        // stages would put a copy and a turn of conversions (1 us) between the end of the previous kernel and the first MMAs.
#pragma unroll
        for (int i = 0; i < kFirst; ++i) {
            const int n = (warp + 16 * i) / MC, t = (warp + 16 * i) % MC;
            if (n < kNB && t < m) {
                int step = step0 + n;
                while (step >= step1) step -= step1 - step0;
                const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
                tc_convert<TYPE, MC, true>(a, first[i], t, step * kTcStepCols, cols_here, b_ring + n * (Shape::kGroupsB * tc_group_b(TYPE)),
                                           info_ring + n * tc_info_floats(TYPE, MC) * 4, n < step1 - step0 ? norm_parts + (n * MC + t) * 4 : 0u, lane);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::bar_arrive(tc::s32(&s_bfull[n]));
            }
        }

        for (int tile = group; tile < n_tiles; tile += n_groups) {
            const int p = part_of(tile), tile0 = first_tile(p);
            const uint32_t mis0 = class_mis(a.part[p], cls);
            const int shift = a.tc_map_shift[p], slot = (((cls & ((1 << shift) - 1)) * 8) >> shift) + (cls >> shift);  // where the class lies
            for (int step = step0; step < step1; ++step) {
                if (!kWide || (st & 1) == pair) {
                    tc::bar_wait(tc::s32(&s_wfull[stage]), wphase, failed);
                    const uint32_t at = stages + stage * kStageBytes, info = info_ring + (st & (kTcInfoSlots - 1)) * tc_info_floats(TYPE, MC) * 4;
                    if constexpr (!kPresplit) {
                        // the warps that share the step take turns at splitting activation rows
                        const int t = kWide ? (warp - (st >> 1) * m) & 7 : (warp - st * m) & 15;
                        if (t < m && st >= kNB) {
                            const int cols_here = a.cols - step * kTcStepCols < kTcStepCols ? a.cols - step * kTcStepCols : kTcStepCols;
                            tc::bar_wait(tc::s32(&s_bempty[bs]), bphase ^ 1u, failed);
                            const uint32_t part = tile == group ? norm_parts + ((step - step0) * MC + t) * 4 : 0u;
                            TcColumns c;
                            const uint32_t xs = at + kTcRows * kPitch + t * (kTcStepCols * 4);
                            int ca, cb;
                            tc_columns<TYPE>(lane, ca, cb);
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(c.v[0]), "=f"(c.v[1]), "=f"(c.v[2]), "=f"(c.v[3]) : "r"(xs + ca * 4));
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(c.v[4]), "=f"(c.v[5]), "=f"(c.v[6]), "=f"(c.v[7]) : "r"(xs + cb * 4));
                            if constexpr (chunk_block(TYPE) < kTcStepCols) {  // (else a step is whole)
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    c.v[i] = ca < cols_here ? c.v[i] : 0.0f;
                                    c.v[4 + i] = cb < cols_here ? c.v[4 + i] : 0.0f;
                                }
                            }
                            tc_convert<TYPE, MC, false>(a, c, t, step * kTcStepCols, cols_here, b_ring + bs * (Shape::kGroupsB * tc_group_b(TYPE)), info, part, lane);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) tc::bar_arrive(tc::s32(&s_bfull[bs]));
                        }
                    }
                    const uint32_t row = at + (slot * 32 + lane) * kPitch + ((mis0 + static_cast<uint32_t>(step) * kStepBytes) & 15u);
                    const uint32_t wempty = tc::s32(&s_wempty[stage]);

                    auto unit = [&](auto odd_tag) {
                        constexpr bool O = decltype(odd_tag)::value != 0;
                        constexpr bool kRowAddress = TYPE == kQ8_0 || TYPE == kIQ4_NL || grid_is_codebook(TYPE);
                        const uint32_t line = kRowAddress ? row : row & (tc_word_loads(TYPE) ? ~3u : ~7u), sh = (row & 2u) * 8u;
                        constexpr int kBC = tc_batch_chunks<TYPE, MC>(), kBatches = tc_half_batches<TYPE, MC>();
                        TcUnit<TYPE> u[tc_halves(TYPE)];
                        [[maybe_unused]] uint32_t ones = 0;
                        auto batch = [&](TcUnit<TYPE> &v, int half, auto batch_tag, bool first_half, bool last_half) {
                            constexpr int B = decltype(batch_tag)::value;
                            const bool first = first_half && B == 0, last = last_half && B == kBatches - 1;
                            if constexpr (tc_signed_table(TYPE)) {
                                constexpr int kCopies = tc_table_copies(TYPE, MC);
                                v.table = table + lane / (32 / kCopies) * 4, v.pitch = 4 * kCopies;
                            } else if constexpr (grid_is_codebook(TYPE)) {
                                v.table = table;
                            }
                            if constexpr (B == 0) v.template begin<O>(line, sh, half);
                            uint32_t r[tc_chunk_regs(TYPE)];
                            v.template chunk<O, B * kBC>(line, sh, half, r);
                            if constexpr (tc_scaled_bytes(TYPE) && !tc_ones_row(TYPE, MC)) {
                                static_assert(kBC == 1, "one chunk at a time");
#pragma unroll
                                for (int i = 0; i < 32; ++i) ones = __dp4a(r[i], 0x01010101u, B == 0 && i == 0 ? 0u : ones);
                            }
                            if (kBC == 1 && last) {  // everything of the stage has been read
                                __syncwarp();
                                if (lane == 0) tc::bar_arrive(wempty);
                            }
                            // the previous batch's MMAs: A may be overwritten, sums are complete
                            tc::bar_wait(mma_done, dphase, failed);
                            dphase ^= 1u;
                            tc::fence_after();
                            tc::st_chunk(tm_mine, r);
                            if ((first || tc_fresh_batches(TYPE)) && pending) tc_accumulate<TYPE, MC>(pend, tm_mine + kTmD, first, unit_sums, acc);
                            if constexpr (kBC == 2) {
                                v.template chunk<O, B * kBC + 1>(line, sh, half, r);
                                if (last) {
                                    __syncwarp();
                                    if (lane == 0) tc::bar_arrive(wempty);
                                }
                                tc::st_chunk(tm_mine + tc_chunk_regs(TYPE), r);
                            }
                            tc::wait_st();
                            tc::fence_before();
                            __syncwarp();
                            if (lane == 0) tc::bar_arrive(a_full);
                            if (last || tc_fresh_batches(TYPE)) {
                                if constexpr (tc_mins(TYPE) > 0) {
#pragma unroll
                                    for (int h = 0; h < tc_halves(TYPE); ++h) pend.unit[h] = u[h];
                                }
                                pend.info = info, pend.kh = kh;
                                if constexpr (tc_scaled_bytes(TYPE) && !tc_ones_row(TYPE, MC)) pend.ones = ones;
                                if constexpr (tc_integer_scale(TYPE)) {
                                    pend.d = v.scale(0);
#pragma unroll
                                    for (int g = 0; g < tc_sums<TYPE, MC>(); ++g) pend.s[g] = __int_as_float(v.integer_scale(2 * B * kBC + g));
                                } else {
#pragma unroll
                                    for (int g = 0; g < tc_sums<TYPE, MC>(); ++g) pend.s[g] = v.scale(tc_block32(TYPE) ? 2 * B * kBC + g : 0);
                                }
                                pending = true;
                            }
                        };
                        auto half_unit = [&](TcUnit<TYPE> &v, int half, bool first, bool last) {
                            batch(v, half, TcInt<0>{}, first, last);
                            if constexpr (kBatches > 1) batch(v, half, TcInt<1>{}, first, last);
                            if constexpr (kBatches > 2) batch(v, half, TcInt<2>{}, first, last), batch(v, half, TcInt<3>{}, first, last);
                            static_assert(kBatches <= 2 || kBatches == 4, "batches of a half");
                        };
                        if constexpr (tc_halves(TYPE) == 1) {
                            half_unit(u[0], kh, true, true);
                        } else {  // (a loop over the halves was measured: smaller code, but 7 % slower)
                            half_unit(u[0], 0, true, false);
                            half_unit(u[1], 1, false, true);
                        }
                    };
                    if constexpr (block_align(TYPE) >= 8 || tc_word_loads(TYPE)) {
                        unit(TcInt<0>{});
                    } else {
                        if (row & 4u) unit(TcInt<1>{});
                        else unit(TcInt<0>{});
                    }
                }
                ++st;
                if (++stage == kStages) stage = 0, wphase ^= 1u;
                if (++bs == kNB) bs = 0, bphase ^= 1u;
            }
            // The next kernel's blocks may come now.  Requested at the start of a block they take the SMs that this grid leaves, and those of its
            // first blocks to end, and hold them until its last one has ended; clusters of the next but one find no room beside them.
            // (With clusters, start of a block and here: the 27B model's pass of 4 rows 5.05 and 4.79 ms, a layer of 1 row on each of three streams
            // 69.5 and 67.0 us, five IQ tensors of 1 row 96.5 and 91.3.  At the start of the last step: 4.81 ms, 68.3 us, 95.3.)
            if (tile + n_groups >= n_tiles) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            // ---- the tile's last sums, then the outputs ----
            unsigned counted = 0;  // thread 0: the column ranges of the tile that are ahead of this one
            if (k_split > 1 && !clustered && threadIdx.x == 0) {
                unsigned *const count = a.partial_counts + (tile - a.tc_first);
                asm volatile("atom.inc.relaxed.gpu.global.u32 %0, [%1], %2;" : "=r"(counted) : "l"(count), "r"(static_cast<unsigned>(k_split) - 1u) : "memory");
            }
            if (pending) {
                tc::bar_wait(mma_done, dphase, failed);
                tc::fence_after();
                tc_accumulate<TYPE, MC>(pend, tm_mine + kTmD, true, unit_sums, acc);
            }
            pending = false;
            tc::fence_before();
            if (tile + n_groups >= n_tiles) asm volatile("bar.arrive 7, %0;" ::"n"(kTcDecoders + 32) : "memory");  // tensor memory may go
            if ((a.fuse & kFuseNorm) && tile == group) {
                tc::decoders_sync();  // (the last squares have been stored)
                if (warp < m) {
                    float sq = 0.0f;
                    for (int i = lane; i < step1 - step0; i += 32) sq += __uint_as_float(lds32(norm_parts + (i * MC + warp) * 4));
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, off);
                    if (!clustered) {
                        if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(tc::s32(&s_norm[0][warp])), "f"(sq) : "memory");
                    } else {
                        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
                        if (lane < k_split) tc::st_async(tc::in_block(tc::s32(&s_norm[rank][warp]), lane), sq, tc::in_block(tc::s32(&s_cluster), lane));
                    }
                }
            }
            float sums[MC];
            acc.get(sums);
            acc.clear();
            if (!clustered) {
                if (k_split > 1 && threadIdx.x == 0) s_count = static_cast<int>(counted);
                tc_finish_tile<TYPE, MC>(a, m, p, tile, tile - tile0, rank, tile + n_groups < n_tiles, red, sums, s_norm[0], &s_count, s_best_v, s_best_i, failed);
                continue;
            }
            // The tile's 256 rows are dealt out to the blocks of the cluster; every block sends each its part of the sums:
            // red[column range][pair of groups][row of the receiver][activation row], counted in bytes on s_cluster
            const int red_rows = a.tc_deal;
            const int r0 = rank * red_rows, r1 = r0 + red_rows < kTcRows ? r0 + red_rows : kTcRows;
#pragma unroll
            for (int round = 0; round < MC / kOut; ++round) {
            {
                const int r = cls + 8 * lane, owner = (r * a.tc_deal_recip) >> 16;
                float out[kOut];
#pragma unroll
                for (int t = 0; t < kOut; ++t) out[t] = sums[round * kOut + t];
                const uint32_t to = red + ((rank * 2 + pair) * red_rows + (r - owner * red_rows)) * (kOut * 4);
                // (once per thread: the cluster's barriers are known to exist)
                if (rounds == 0 && !((a.fuse & kFuseNorm) && warp < m)) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
                if (threadIdx.x == 0) {
                    const int bytes = (r1 - r0) * (2 * kOut * 4) * k_split + ((a.fuse & kFuseNorm) && tile == group ? m * k_split * 4 : 0);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::s32(&s_cluster)), "r"(bytes) : "memory");
                }
                tc::st_async_row<kOut>(tc::in_block(to, owner), out, tc::in_block(tc::s32(&s_cluster), owner));
            }
            tc::bar_wait_cluster(tc::s32(&s_cluster), rounds & 1u, failed);
            {
                const int t = round * kOut + (warp & (kOut - 1));
                const MatvecPart &part = a.part[p];
                if (t < m) {
                    float factor = 1.0f;
                    if (a.fuse & kFuseNorm) {
                        float sq = 0.0f;
                        for (int k = 0; k < k_split; ++k) sq += s_norm[k][t];
                        factor = 1.0f / sqrtf(sq / static_cast<float>(a.cols) + a.eps);
                    }
                    for (int r = r0 + (warp / kOut) * 32; r < r1; r += 512 / kOut) {
                        const int row = (tile - tile0) * kTcRows + r + lane;
                        const bool exists = r + lane < r1 && row < part.rows;
                        float sum = 0.0f;
                        if (exists) {
#pragma unroll
                            for (int k = 0; k < kMaxSplit; ++k)
                                if (k < k_split) {
                                    const uint32_t at = red + ((2 * k * red_rows + (r + lane - r0)) * kOut + (warp & (kOut - 1))) * 4;
                                    sum += __uint_as_float(lds32(at)) + __uint_as_float(lds32(at + kOut * red_rows * 4));
                                }
                            sum = tc_put<TYPE>(a, part, row, t, sum, factor);
                        }
                        if (a.out_idx != nullptr) tc_note_best(exists, sum, row, lane, &s_best_v[warp][t], &s_best_i[warp][t]);
                    }
                }
            }
            if (round + 1 < MC / kOut || tile + n_groups < n_tiles) {  // the sums may be overwritten once everybody has read them
                tc::decoders_sync();
                if (threadIdx.x < static_cast<unsigned>(k_split))
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tc::in_block(tc::s32(&s_read), threadIdx.x))
                                 : "memory");
                tc::bar_wait_cluster(tc::s32(&s_read), rounds & 1u, failed);
            }
            ++rounds;
            }
        }
    }
    if (clustered && warp >= 16) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // (every thread takes part)
    if (lane == 0 && *failed) atomicCAS(a.status, 0u, kStatusWaitExpired);
    if (a.out_idx != nullptr) tc_finish_argmax(a, m, warp, lane, s_best_v, s_best_i, &s_last);
}

}  // namespace vqm
