// Quantized matvec for 1..24 activation rows on the 5th-generation tensor cores:  y[t][r] = sum_k W[r][k] x[t][k].
//
// Same contract as the CUDA-core kernel (vqm_matvec.cuh): raw GGUF blocks read once for all activation rows, inputs and
// sums of fp32 precision.  What bounds that kernel is instruction issue - a permute, half a packed FMA and half a packed
// FMA per activation row for every weight - so here the multiplications go to tcgen05.mma and a thread only unpacks:
//   * The integer part of a weight (quant, or quant times its integer sub-scale: at most 11 significant bits) is exact in
//     fp16.  Quants are masked out of the raw words two at a time and ARE fp16 subnormals (q * 2^-24), one LOP3 per two
//     weights; one packed fp16 multiply (or FMA, for a bias) makes them (q - bias) * sub-scale * 2^-24, exactly.  fp16
//     super-scales stay outside: the sums of a unit of columns are multiplied by them in fp32.
//   * An activation is split exactly into three fp16 values, x = s * (h0 + 2^-11 h1 + 2^-22 h2), s a power of two chosen
//     per 256 columns (33 bits for a 24-bit number; values below the chunk's largest lose nothing either until they
//     are 2^-32 of it).  The planes are separate columns of the B operand, so M rows make 3M columns.  Products are exact,
//     the tensor core adds in fp32.
//     Q3_K and Q2_K: quant times sub-scale fits into 8 bits, and everything is a byte and an integer: a quarter of the multiplies
//     that scale, half the stores to tensor memory, exact sums (see TcUnit<kQ3_K>, tc_convert_bytes).  Q8_0, IQ4_NL and IQ4_XS: the
//     weight without its scale is a byte already, and each block of 32 has its own sum.  An activation is six bytes then.
//   * A block owns 256 rows.  Thread = weight row (lane of tensor memory): scales are decoded once per row, by the one
//     thread that needs them, and the A operand is written from registers to tensor memory with tcgen05.st (measured: an
//     MMA of 128 x 16 with A in tensor memory takes 9.4 cycles at N = 16 and 16.4 at N = 32; with A in shared memory 40).
//
// A block: 16 decoder warps in four groups, one copy warp and two warps that issue the MMAs of two groups each.  Two groups
// share the 256 rows of a step (a superblock column of 256); the two pairs take the steps in turn, or half of the columns of
// each (tc_wide).
//   copy warp    one to eight TMA tile copies (the row classes below) and one bulk copy per activation row into
//                the stage ring;
//   converters   the decoder warps take turns to split one activation row's 256 columns into the B operand (shared memory);
//   decoders     raw words -> 64 A columns at a time (a "chunk": 32 tensor-memory columns), two chunks to a batch of
//                eight MMAs.  The first chunk of the next batch is decoded into registers while the MMAs run; then it is
//                stored and, at the end of a unit, the sums are read back with tcgen05.ld.
// (Letting the last decoder warp to arrive issue the MMAs and the copies instead of separate warps was measured: 20 % slower,
// the late warp of a group becomes later.)
// Rows are dealt to warps by class: warp c (of 8) holds rows c, c + 8, ... of the block's 256.  Blocks of most types are
// only 2-byte aligned; 8 rows further the position within a 16-byte line repeats, so all lanes of a warp see the same
// misalignment, and tile copies of 32 rows of a class have a 16-byte aligned row stride.  The stage's row pitch is an odd
// multiple of 16 bytes, free of bank conflicts for 16-byte loads.
//
// Columns are split over k_split blocks, each a contiguous range of steps.  The blocks exchange their sums through memory (tc_finish_tile) or,
// where the launch has been given no room for them (a captured graph, a caller without a runtime, a stream alone on the GPU), as a cluster: a tile's rows are dealt out to its blocks
// and every block sends each its part (st.async).  Both add the parts in the order of the columns: the split and the order of all additions depend
// on rows and columns only, never on M.
#pragma once

#include <cuda.h>

#include "vqm_formats.cuh"
#include "vqm_kernels.h"
#include "vqm_steps.cuh"

namespace vqm {

// (608 threads cap every thread at 96 registers.  The 16-row kernels of Q4_K, Q5_K, Q6_K and Q2_K spill 8 to 44 bytes, all 24-row kernels 8 to 52.)
constexpr int kTcRows = kTcTileRows, kTcStepCols = 256, kTcDecoders = 512, kTcThreads = kTcDecoders + 96;
constexpr int kTcCore = 144;                      // bytes from one 8-column core matrix of B to the next (128 + 16: no bank conflicts)
constexpr int kTcInfoSlots = 8;                   // ring of per-step activation scales and group sums
constexpr int kTcMaxNormSteps = 128;
constexpr int kTcElemBytes = 2;                   // element of the tensor maps (rows are even numbers of bytes)

// ---- per-type constants ------------------------------------------------------------------------------------------------
__host__ __device__ constexpr int tc_step_bytes(int type) { return kTcStepCols / chunk_block(type) * chunk_block_bytes(type); }
// pitch of a row in a stage: the step's bytes behind up to 14 bytes of misalignment, an odd multiple of 16
__host__ __device__ constexpr int tc_pitch(int type) {
    const int lines = (tc_step_bytes(type) + (block_align(type) >= 16 ? 0 : 16 - block_align(type)) + 15) / 16;
    return (lines | 1) * 16;
}
// Rows that are not 8-byte aligned are read either in 8-byte loads, by one of two copies of the decoder (rows that start in the
// lower and in the upper word), or in 4-byte loads, which have twice the bank conflicts.  As fp16, Q3_K 75776 x 5120, 1 row: 74 us with
// two copies (they do not fit into the instruction cache), 64 us with word loads; Q6_K, which loads twice as much: 84 and 88.
__host__ __device__ constexpr bool tc_word_loads(int type) { return block_align(type) < 8 && type != kQ6_K; }
// A columns per weight: 2 where quant times sub-scale needs more than 11 bits and is split in two
__host__ __device__ constexpr int tc_parts(int type) { return type == kQ6_K ? 2 : 1; }
// types that look up four signed weights at a time (see TcSigned)
__host__ __device__ constexpr bool tc_signed_table(int type) { return type == kIQ2_XXS || type == kIQ3_XXS || type == kIQ3_S; }
// Copies of the signed table, word by word: 32 lanes that pick words at random from 32 banks take 3.5 turns, 16 from every other bank 3.1,
// 8 from every fourth 2.6.  As many as there is room for.
__host__ __device__ constexpr int tc_table_copies(int type, int mc) {
    return type == kIQ3_XXS ? (mc <= 4 ? 4 : 2) : type == kIQ2_XXS ? 2 : type == kIQ3_S && mc <= 4 ? 2 : 1;
}
__host__ __device__ constexpr int tc_table_bytes(int type, int mc) {
    return tc_signed_table(type) ? (type == kIQ3_XXS ? 16384 : 32768) * tc_table_copies(type, mc) : grid_bytes(type);
}
// types whose scale covers 32 weights and stays outside: a sum per 32 columns instead of one per unit; with an integer scale the sums
// (of the larger part of the activations) stay integers until the super-scale
__host__ __device__ constexpr bool tc_block32(int type) { return type == kQ8_0 || type == kIQ4_NL || type == kIQ4_XS; }
__host__ __device__ constexpr bool tc_integer_scale(int type) { return type == kIQ4_XS; }
__host__ __device__ constexpr int tc_groups(int type) { return type == kQ4_K || type == kQ5_K ? 8 : type == kQ2_K ? 16 : 0; }  // minimums per step
// Types whose weights times sub-scale fit into 8 bits (see TcUnit<kQ3_K>; a step is one unit) ...
__host__ __device__ constexpr bool tc_scaled_bytes(int type) { return type == kQ3_K || type == kQ2_K; }
__host__ __device__ constexpr int tc_byte_offset(int type) { return type == kQ3_K ? 127 : 0; }  // what an A byte is above the weight
// ... and types whose weights themselves are bytes (signed ones): their operands are bytes (kind::i8).
__host__ __device__ constexpr bool tc_bytes(int type) { return tc_scaled_bytes(type) || tc_block32(type); }
__host__ __device__ constexpr int tc_mins(int type) { return tc_scaled_bytes(type) ? tc_groups(type) : tc_groups(type) / 2; }  // per half (whole) step
__host__ __device__ constexpr int tc_group_b(int type) { return (tc_bytes(type) ? 16 : 32) * kTcCore; }  // bytes of 8 B rows over a step
__host__ __device__ constexpr int tc_chunk_regs(int type) { return tc_block32(type) ? 16 : 32; }  // tensor-memory columns of a chunk
// order of a B core row's 8 columns, made of the column words a and b (4 columns each), see tc_columns
enum : int { kOrderNibbles = 0, kOrderBytes = 1, kOrderGrid = 2 };
__host__ __device__ constexpr int tc_order(int type) {
    return grid_is_codebook(type) ? kOrderGrid : (type == kIQ4_NL || type == kIQ4_XS) ? kOrderBytes : kOrderNibbles;
}
// log2 of the number of tensor maps of a weight tensor (vqm_tcmv_maps.cu): its row classes share 1, 2, 4 or 8
inline int tc_map_shift(int rows, long long row_bytes) {
    return rows % 8 != 0 ? 3 : row_bytes % 16 == 0 ? 0 : row_bytes % 8 == 0 ? 1 : row_bytes % 4 == 0 ? 2 : 3;
}
struct TcMaps1 {
    CUtensorMap m[1][8];
};
struct TcMaps4 {
    CUtensorMap m[kMaxParts][8];
};

// cuTensorMapEncodeTiled of the driver (vqm_tcmv_maps.cu)
using TcEncode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                              const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
cudaError_t tc_encoder(TcEncode *out);

// Which part of a step a warp group takes: whole steps, every other one (wide types), or half of the columns of every step
// where two steps of weights in use and one in flight do not fit into shared memory.
__host__ __device__ constexpr bool tc_wide(int type) { return tc_pitch(type) <= 176; }

constexpr int kTcPlanes = 6;  // of activations as bytes
// bits of their first two planes: with an integer scale the sums of a superblock must fit into 32 bits
__host__ __device__ constexpr int tc_piece_bits(int type) { return tc_integer_scale(type) ? 11 : 14; }
// (16 rows of scaled bytes fill a group's tensor memory; the decoders add their bytes up themselves then.)
__host__ __device__ constexpr bool tc_ones_row(int type, int mc) { return tc_scaled_bytes(type) && mc <= 8; }
// activation rows a kernel is compiled for, their B rows (3 planes; bytes: 6 planes, unsigned ones a row of ones too) in groups of 8, and
// the MMA's N
template <int TYPE, int MC>
struct TcShape {
    static constexpr int kRowsB = tc_bytes(TYPE) ? kTcPlanes * MC + (tc_ones_row(TYPE, MC) ? 1 : 0) : 3 * MC;
    static constexpr int kGroupsB = (kRowsB + 7) / 8;
    static constexpr int kN = (kGroupsB + 1) / 2 * 16;
};
// per step: the activation rows' scales (bytes with an offset: and three integer sums each), then the sums of the column groups that share a minimum
__host__ __device__ constexpr int tc_info_rows(int mc) { return mc < 4 ? 4 : mc; }
__host__ __device__ constexpr int tc_info_scales(int type, int mc) { return (tc_byte_offset(type) != 0 ? 4 : 1) * tc_info_rows(mc); }
__host__ __device__ constexpr int tc_info_floats(int type, int mc) { return tc_info_scales(type, mc) + tc_groups(type) * mc; }
// More than 8 activation rows: their B operand and infos come ready-made (tc_split_kernel), by bulk copies, because the stages
// have no room for 16 KB of activations; the tile's sums go out 8 (of 24: 4) activation rows at a time.
__host__ __device__ constexpr bool tc_presplit(int mc) { return mc > 8; }
__host__ __device__ constexpr int tc_out_rows(int mc) { return mc > 16 ? 4 : mc > 8 ? 8 : mc; }
// pitch of the sums of a tile's rows in shared memory (tc_red_at; the parts of a cluster's blocks take at most 264 rows)
constexpr int kTcRedRows = kTcRows + kTcRows / 8;
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_stage_bytes() { return kTcRows * tc_pitch(TYPE) + (tc_presplit(MC) ? 0 : MC * kTcStepCols * 4); }
// Shared memory beside the weight stages, with `b` B stages (an MMA may read one group of rows further).
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_fixed_bytes(int b) {
    return (tc_table_bytes(TYPE, MC) + 127) / 128 * 128 + (b * TcShape<TYPE, MC>::kGroupsB + 1) * tc_group_b(TYPE) + kTcInfoSlots * tc_info_floats(TYPE, MC) * 4 +
           2 * kTcRedRows * tc_out_rows(MC) * 4 + (tc_presplit(MC) ? 0 : (kTcMaxNormSteps + 2) * MC * 4) + 256;
}
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_stages_beside(int b) {
    const int s = (226 * 1024 - 1024 - tc_fixed_bytes<TYPE, MC>(b)) / tc_stage_bytes<TYPE, MC>();
    return s > 6 ? 6 : s;  // (the info ring must have two slots more)
}
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_b_stages() { return tc_stages_beside<TYPE, MC>(4) >= 4 ? 4 : tc_stages_beside<TYPE, MC>(3) >= 3 ? 3 : 2; }
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_stages() { return tc_stages_beside<TYPE, MC>(tc_b_stages<TYPE, MC>()); }
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_smem_bytes() {
    return 1024 + tc_fixed_bytes<TYPE, MC>(tc_b_stages<TYPE, MC>()) + tc_stages<TYPE, MC>() * tc_stage_bytes<TYPE, MC>();
}

// bytes of a step in the buffer of ready-made B operands: the operand, then the infos
template <int TYPE, int MC>
__host__ __device__ constexpr int tc_split_bytes() { return TcShape<TYPE, MC>::kGroupsB * tc_group_b(TYPE) + tc_info_floats(TYPE, MC) * 4; }
// 16 activation rows at a time: not the types with a sum per 32 columns (192 columns of sums do not fit beside A in tensor memory)
__host__ __device__ constexpr bool tc_sixteen(int type) { return !tc_block32(type); }
// 24 at a time: where their sums fit into a group's tensor memory (not six planes) and their B operands leave room for the stages
template <int TYPE>
__host__ __device__ constexpr bool tc_twenty_four() { return tc_sixteen(TYPE) && !tc_bytes(TYPE) && tc_stages_beside<TYPE, 24>(2) >= (tc_wide(TYPE) ? 3 : 2); }

// ---- primitives --------------------------------------------------------------------------------------------------------
namespace tc {
__device__ __forceinline__ uint32_t s32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool bar_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits are bounded (two seconds by the global timer).  Once one wait of the block has run out (`failed`) the others give up
// at once and everybody runs through to the end: results are garbage, the status word says so, nothing hangs.
static __device__ __noinline__ bool give_up(unsigned long long *began, volatile int *failed) {
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (*began == 0) *began = now;
    if (now - *began > 2000000000ull) *failed = 1;
    return *failed != 0;
}
// (A form with a vote, so that the branches are uniform and need no reconvergence code, was measured: 8 % slower kernels.  It
// polls faster, and polls of one warp delay the barriers of the others.)
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, volatile int *failed) {
    if (bar_try(bar, parity)) return;
    unsigned long long began = 0;
#pragma unroll 1
    for (uint32_t i = 1;; ++i) {
        if (bar_try(bar, parity)) return;
        if ((i & 255u) == 0 && give_up(&began, failed)) return;
    }
}
// acquire at cluster scope, for what other blocks of the cluster have stored
__device__ __forceinline__ void bar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *failed) {
    if (bar_try_cluster(bar, parity)) return;
    unsigned long long began = 0;
#pragma unroll 1
    for (uint32_t i = 1;; ++i) {
        if (bar_try_cluster(bar, parity)) return;
        if ((i & 255u) == 0 && give_up(&began, failed)) return;
    }
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D (tensor memory) (+)= A (tensor memory, 128 x 32 bytes) * B (shared memory, N x 32 bytes, K-major core matrices); 16 fp16 or
// 32 bytes along K, sums in fp32 or 32-bit integers
template <int TYPE>
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if constexpr (tc_bytes(TYPE)) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// Instruction descriptor: 128 rows, N columns; fp32 += fp16 * fp16, s32 += u8 * u8 or s32 += s8 * s8.
__host__ __device__ constexpr uint32_t instruction(int type, int n) {
    return ((tc_bytes(type) ? 2u : 1u) << 4) | (tc_bytes(type) && !tc_scaled_bytes(type) ? (1u << 7) | (1u << 10) : 0u) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}
// Shared-memory descriptor without swizzle: 8 x 16-byte core matrices, kTcCore bytes apart along K, tc_group_b bytes along N.
template <int TYPE>
__device__ __forceinline__ uint64_t b_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(kTcCore >> 4) << 16) |
           (static_cast<uint64_t>(tc_group_b(TYPE) >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void st32(uint32_t at, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(at),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void ld4(uint32_t at, float *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void st16(uint32_t at, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(at),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void st_chunk(uint32_t at, const uint32_t (&r)[32]) { st32(at, r); }
__device__ __forceinline__ void st_chunk(uint32_t at, const uint32_t (&r)[16]) { st16(at, r); }
__device__ __forceinline__ void ld1(uint32_t at, uint32_t &v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(at) : "memory");
}
__device__ __forceinline__ void ld4(uint32_t at, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ld8(uint32_t at, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(at)
                 : "memory");
}
__device__ __forceinline__ void ld8(uint32_t at, float *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(at)
                 : "memory");
}
// the 3 * MC sums of this thread's row
template <int MC>
__device__ __forceinline__ void ld_sums(uint32_t at, float (&v)[3 * MC + 1]) {
    if constexpr (MC == 1) {
        ld4(at, v);
    } else {
        float w[(3 * MC + 7) / 8 * 8];
#pragma unroll
        for (int i = 0; i < (3 * MC + 7) / 8; ++i) {
            if (i * 8 + 4 >= 3 * MC) ld4(at + i * 8, w + i * 8);
            else ld8(at + i * 8, w + i * 8);
        }
#pragma unroll
        for (int i = 0; i < 3 * MC; ++i) v[i] = w[i];
    }
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void decoders_sync() { asm volatile("bar.sync 5, 512;" ::: "memory"); }
// the address, in the cluster's shared window, of the same variable in block `rank`
__device__ __forceinline__ uint32_t in_block(uint32_t local, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// stores into another block's shared memory that count their bytes on that block's barrier
__device__ __forceinline__ void st_async(uint32_t at, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(at), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
template <int MC>
__device__ __forceinline__ void st_async_row(uint32_t at, const float (&v)[MC], uint32_t bar) {
    if constexpr (MC == 1) {
        st_async(at, v[0], bar);
    } else if constexpr (MC == 2) {
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(at), "r"(__float_as_uint(v[0])),
                     "r"(__float_as_uint(v[1])), "r"(bar)
                     : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < MC; i += 4)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(at + i * 4),
                         "r"(__float_as_uint(v[i])), "r"(__float_as_uint(v[i + 1])), "r"(__float_as_uint(v[i + 2])), "r"(__float_as_uint(v[i + 3])),
                         "r"(bar)
                         : "memory");
    }
}

// packed fp16 arithmetic on raw words
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// Byte K of `w` twice, as fp16 `base + byte * 2^-s` (hi: the upper byte of fp16 `base` four times; the byte is its mantissa's low end).
template <int K>
__device__ __forceinline__ uint32_t byte_h2(uint32_t w, uint32_t hi) { return __byte_perm(w, hi, 0x4040 | (K << 8) | K); }
constexpr uint32_t kHi1024 = 0x64646464u, kHi64 = 0x54545454u;  // 1024 + b, 64 + b / 16

// ---- raw words of a row -------------------------------------------------------------------------------------------------
// N consecutive 32-bit words at byte OFF (a multiple of 4) behind the row's first byte.  `line` is the row's address rounded
// down to 8 (4 with word loads); O says whether the row starts in the upper word there, `sh` is 16 if it starts in the middle of
// a word.
template <int TYPE, bool O, int OFF, int N>
__device__ __forceinline__ void words(uint32_t line, uint32_t sh, uint32_t (&w)[N]) {
    constexpr int A = block_align(TYPE);
    if constexpr (A >= 16 && OFF % 16 == 0 && N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const uint4 v = lds128u(line + OFF + 16 * i);
            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
        }
    } else if constexpr (tc_word_loads(TYPE)) {
        constexpr bool kShift = A < 4;
        uint32_t r[N + 1];
#pragma unroll
        for (int i = 0; i < N + (kShift ? 1 : 0); ++i) r[i] = lds32(line + OFF + 4 * i);
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = kShift ? __funnelshift_r(r[i], r[i + 1], sh) : r[i];
    } else {
        constexpr int first = (OFF / 4) % 2 + (O ? 1 : 0);  // word of the first 8-byte load that holds word 0
        constexpr int skip = first >= 2 ? 8 : 0, lead = first % 2;
        constexpr bool kShift = A < 4;
        constexpr int need = lead + N + (kShift ? 1 : 0), loads = (need + 1) / 2;
        uint32_t r[2 * loads];
#pragma unroll
        for (int i = 0; i < loads; ++i) {
            const unsigned long long v = lds64(line + OFF / 8 * 8 + skip + 8 * i);
            r[2 * i] = static_cast<uint32_t>(v), r[2 * i + 1] = static_cast<uint32_t>(v >> 32);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if constexpr (kShift) w[i] = __funnelshift_r(r[lead + i], r[lead + i + 1], sh);
            else w[i] = r[lead + i];
        }
    }
}
}  // namespace tc
}  // namespace vqm
