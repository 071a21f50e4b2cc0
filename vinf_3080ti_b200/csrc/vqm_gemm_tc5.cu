// Prompt-pass GEMM on the 5th-generation tensor cores:  Y[t][r] = sum_k W[r][k] X[t][k]  for hundreds of activation rows.
//
// Same contract as the warp-level kernel in vqm_gemm.cu (replaces the reference's vinf_qgemm_kernel,
// engine/csrc/megakernel/qwen_runtime.cu:655-769: fp16 operands, fp32 accumulation), built on tcgen05:
//   * two blocks of a cluster (two SMs) work as a pair on tcgen05.mma.cta_group::2: 256 weight rows (128 decoded by each
//     block) by NH accumulators of up to 256 activation rows, half of which each block holds in its shared memory.  The
//     first block issues the MMAs for both and commits to the barriers of both (multicast commit), the second forwards its
//     "full" stages with one remote arrive each, each block drains its own 128 lanes of tensor memory;
//   * K is walked in stages of 64 columns, as many stage buffers as fit;
//   * one thread of warp 18 brings the raw weight bytes, 256 columns ("a run") of the block's rows at a time, into a ring of
//     buffers by TMA tile copies (by row class, see vqm_tcmv_maps.cu; a bulk copy per row takes the copy unit 33 cycles, 98
//     instead of 76 us for 64 activation rows x 17408 x 5120).  F16 and F32, whose runs are too wide for the ring, are
//     decoded straight from global memory;
//   * warps 0-15 dequantise: two or four groups of warps take the stages in turn, thread = weight row, so that scales
//     are unpacked once per 32 weights and a warp does one wait, one fence and one arrive per 1024 or 2048 weights.  The weights are
//     decoded into registers before the wait for the stage, which is then held for eight stores per thread only;
//   * one thread of warp 16 feeds the activations, one TMA tile copy per stage and accumulator (no multicast);
//   * one thread of warp 17 issues, per stage, 4 K-steps x NH tcgen05.mma (kind::f16) and commits them to "empty";
//   * after the last commit, warps 0-15 read the accumulators with tcgen05.ld and store y, 32 consecutive rows per warp.
//
// What bounds it: with 512 activation rows the MMAs (0.60 us per stage alone, 0.75 on the whole GPU under the power cap), up
// to 256 the decoders (0.39 us per stage).  Before, four threads shared a row and a stage was handed over as two halves with a
// wait, fence, arrive and commit each, from a lane that the compiler could not tell to be alone (see elect_one): 0.36 us per
// half before any weight was decoded.  64 / 256 / 512 rows: Q4_K 17408 x 5120 79 / 81 / 92 us before, 42 / 48 / 72 now; Q6_K
// 6144 x 5120 77 / 77 / 89 and 27 / 31 / 44, Q4_K 5120 x 17408 236 / 237 / 271 and 49 / 57 / 84 (columns split).
//
// Split of the columns: tensors of few rows leave most SMs idle (6144 rows x 512: 24 pairs of 74), so up to four pairs form
// a cluster that shares the columns of 256 weight rows.  Each pair sums its own range of columns; then every pair sends the
// others their parts of its sums through distributed shared memory and adds what it receives in the order of the columns.
// Every mbarrier wait is bounded: on expiry the block records a status code, everybody falls through to the end, and
// the tensor memory is released before the block returns.
#include <cuda.h>  // CUtensorMap (types only; nothing links against the driver)
#include <cuda_fp16.h>

#include "vqm_formats.cuh"
#include "vqm_kernels.h"
#include "vqm_steps_iq4.cuh"
#include "vqm_tcmv.cuh"

namespace vqm {
namespace {

// Activation rows of an accumulator: up to 256, a multiple of 64 (the MMA's N); NH accumulators: 1 or 2 (512 columns of
// tensor memory, the whole of an SM's: one block per SM).
constexpr int kTM = 128, kTNMax = 256, kTK = 64, kMaxPairs = 4;
constexpr int kMaxStages = 6;
constexpr int kTA = kTM * kTK * 2, kTB = kTNMax / 2 * kTK * 2;  // 16 KB of a block's weights, 16 KB of its half of the activations
constexpr int kAThreads = 512;             // decoder warps 0-15
constexpr int kTThreads = kAThreads + 96;  // warp 16: activation tiles; warp 17: MMAs; warp 18: raw weights
// Raw-block ring: a "run" is 256 weight columns of the 128 rows; a row's bytes of one run are contiguous.
constexpr int kRawCols = 256, kStagesPerRun = kRawCols / kTK;
__host__ __device__ constexpr int raw_run_bytes(int type) { return kRawCols / chunk_block(type) * chunk_block_bytes(type); }
__host__ __device__ constexpr int raw_pitch(int type) { return tc_pitch(type); }  // bytes of a row in a buffer
// (Q8_0, whose buffers are the largest, has two: three leave room for two stages of weights.  17408 x 5120, 64 and 256 rows: 53 and 61 us, 48 and
// 56 so.)
__host__ __device__ constexpr int raw_buffers(int type, int nh) { return nh == 1 && raw_pitch(type) < 256 ? 3 : 2; }
__host__ __device__ constexpr int table_bytes16(int type) { return grid_bytes(type) > 0 ? (grid_bytes(type) + 15) / 16 * 16 : 16; }
__host__ __device__ constexpr bool raw_staged(int type) { return raw_run_bytes(type) <= 288; }  // every quantised type
__host__ __device__ constexpr int raw_ring_bytes(int type, int nh) { return raw_staged(type) ? raw_buffers(type, nh) * kTM * raw_pitch(type) + 16 : 0; }
// Activation tiles in flight (32 KB each in blocks of two accumulators), and as many weight tiles as fit beside them.
__host__ __device__ constexpr int x_stages(int nh) { return nh == 1 ? 4 : 3; }
__host__ __device__ constexpr int tc5_smem_bytes(int type, int nh, int stages) {
    return table_bytes16(type) + 1024 + x_stages(nh) * nh * kTB + stages * kTA + raw_ring_bytes(type, nh);
}
__host__ __device__ constexpr int stages_for(int type, int nh) {
    int s = kMaxStages;
    while (s > 2 && tc5_smem_bytes(type, nh, s) > 226 * 1024) --s;
    return s;
}
// Exchange between the pairs of a cluster: per accumulator, chunks of 16 activation rows go to pair (chunk % pairs), which
// keeps the other pairs' sums of its chunks, 8 KB each, where the stages were.
constexpr int kXChunk = 16, kXBytes = kXChunk * kTM * 4;

using tc::bar_arrive, tc::bar_init, tc::bar_try, tc::bar_try_cluster, tc::in_block, tc::s32;
// Bounded wait; also gives up as soon as another thread of the block has (`failed` is a shared flag).
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int *failed) {
#pragma unroll 1
    for (int i = 0; i < (1 << 22); ++i) {  // a second or so
        // plain try_wait: measured against a suspend-time hint of 2 us (4 us slower on 125) and a test_wait spin (6 us slower)
        if (bar_try(bar, parity)) return true;
        if (*failed) return false;
        if (i > 4096) __nanosleep(200);  // only a wait that is already far beyond a pipeline step backs off
    }
    *failed = 1;
    return false;
}
__device__ __forceinline__ bool bar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *failed) {
#pragma unroll 1
    for (int i = 0; i < (1 << 22); ++i) {
        if (bar_try_cluster(bar, parity)) return true;
        if (*failed) return false;
        if (i > 4096) __nanosleep(200);
    }
    *failed = 1;
    return false;
}

// Warp-wide forms (every lane of the warp calls them together).
//   warp_wait: every lane polls and the warp votes, so that it takes one branch even when a wait gives up.  (Polling by
//              lane 0 alone with a broadcast was measured: slower, 204 instead of 141 us for Q4_K 17408 x 5120 x 512.)
//   warp_arrive: one arrive per warp instead of 32 atomics on the barrier word, after the warp's own writes (and proxy
//              fences); __syncwarp orders them before lane 0's arrive.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *failed) {
    return __all_sync(0xFFFFFFFFu, bar_wait(bar, parity, failed) ? 1 : 0) != 0;
}
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) bar_arrive(bar);
}

// Shared-memory matrix descriptor of a K-major tile in the 128-byte swizzle: rows of 64 fp16 = 128 bytes, groups of 8
// rows 1024 bytes apart (stride byte offset), tile base 1024-byte aligned; version 1 (sm_100), layout type 2.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}
// ---- slot decoders ---------------------------------------------------------------------------------------------------
// N * 32 weights of one row, columns 32 G .. of a 256-column run at `blk` (shared memory), as 16 N words `h` of two fp16
// (N = 1, or N = 2 and G even: what two neighbouring slots share is read once).
// Every value is the fp32 expression of deq8 rounded once to fp16, whichever decoder produces it.  G is a run-time value
// (uniform over the warp): one copy of the code for all slots stays in the instruction cache.
__device__ __forceinline__ uint32_t f16x2_of(f32x2 v) {  // (lo, hi) -> two fp16 in one word, round to nearest even
    float lo, hi;
    unpack2(v, lo, hi);
    uint32_t h;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(hi), "f"(lo));
    return h;
}
// the four bytes of `w` times dl plus nml (packed), as fp16
__device__ __forceinline__ void bytes_fma_f16(uint32_t w, f32x2 neg_magic, f32x2 dl, f32x2 nml, uint32_t &h0, uint32_t &h1) {
    h0 = f16x2_of(fma2(bytes_to_pair<0, 1>(w, neg_magic), dl, nml));
    h1 = f16x2_of(fma2(bytes_to_pair<2, 3>(w, neg_magic), dl, nml));
}
// the four bytes of `w` (minus the bias inside neg_magic) times dl (packed), as fp16
__device__ __forceinline__ void bytes_mul_f16(uint32_t w, f32x2 neg_magic, f32x2 dl, uint32_t &h0, uint32_t &h1) {
    h0 = f16x2_of(mul2(bytes_to_pair<0, 1>(w, neg_magic), dl));
    h1 = f16x2_of(mul2(bytes_to_pair<2, 3>(w, neg_magic), dl));
}
// N words at a 2-byte aligned address
template <int N>
__device__ __forceinline__ void words_a2(uint32_t at, uint32_t (&w)[N]) {
    const uint32_t base = at & ~3u, sh = (at & 2u) * 8u;
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) r[i] = lds32(base + 4 * i);
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(r[i], r[i + 1], sh);
}

template <int TYPE, int N>
__device__ __forceinline__ void decode_slots(uint32_t blk, int G, const uint8_t *table, uint32_t (&h)[16 * N]) {
    if constexpr (TYPE == kQ4_K || TYPE == kQ5_K) {
        // d, dmin, 12 bytes of 6-bit scales and minimums; slot G is sub-block G: d * sc * q - dmin * mn (16-byte aligned blocks)
        const uint4 hd = lds128u(blk);
        const uint32_t qa = blk + (TYPE == kQ4_K ? 16 : 48) + 32 * (G >> 1);
        const uint4 q0 = lds128u(qa), q1 = lds128u(qa + 16);
        const uint32_t q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        uint32_t f[8];
        if constexpr (TYPE == kQ5_K) {
            const uint4 f0 = lds128u(blk + 16), f1 = lds128u(blk + 32);
            f[0] = f0.x, f[1] = f0.y, f[2] = f0.z, f[3] = f0.w, f[4] = f1.x, f[5] = f1.y, f[6] = f1.z, f[7] = f1.w;
        }
        const f32x2 neg_magic = pack2(-8388608.0f, -8388608.0f);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int g = G + k, s = 8 * (g & 3), sh = N == 2 ? 4 * k : 4 * (g & 1);
            const uint32_t y = hd.y >> s, z = hd.z >> s, w3 = hd.w >> s;
            const uint32_t sc = g < 4 ? y & 63u : (w3 & 15u) | ((y >> 2) & 48u), mn = g < 4 ? z & 63u : ((w3 >> 4) & 15u) | ((z >> 2) & 48u);
            const float dl = half_bits_to_float(hd.x & 0xFFFFu) * static_cast<float>(sc);
            const float nml = -half_bits_to_float(hd.x >> 16) * static_cast<float>(mn);
            const f32x2 dl2 = pack2(dl, dl), nml2 = pack2(nml, nml);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint32_t w = (q[i] >> sh) & 0x0F0F0F0Fu;
                if constexpr (TYPE == kQ5_K) w += ((f[i] >> g) & 0x01010101u) * 16u;
                bytes_fma_f16(w, neg_magic, dl2, nml2, h[16 * k + 2 * i], h[16 * k + 2 * i + 1]);
            }
        }
    } else if constexpr (TYPE == kQ6_K) {
        // low nibbles @0, high bit pairs @128, int8 scales @192 (per 16 columns), d @208: d * sc * (q - 32)
        const int n = G >> 2;
        uint32_t hi[8];
        words_a2<8>(blk + 128 + 32 * n, hi);
        const float d = half_bits_to_float(lds16(blk + 208));
        const f32x2 neg_magic = pack2(-(8388608.0f + 32.0f), -(8388608.0f + 32.0f));
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int j = (G & 3) + k, ls = (j >> 1) * 4, hs = 2 * j;
            uint32_t lo[8];
            words_a2<8>(blk + 64 * n + 32 * (j & 1), lo);
            const uint32_t sc = lds16(blk + 192 + 2 * (G + k));
            const float dl[2] = {d * static_cast<float>(static_cast<int8_t>(sc & 0xFFu)), d * static_cast<float>(static_cast<int8_t>(sc >> 8))};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t q = ((lo[i] >> ls) & 0x0F0F0F0Fu) + ((hi[i] >> hs) & 0x03030303u) * 16u;
                bytes_mul_f16(q, neg_magic, pack2(dl[i >> 2], dl[i >> 2]), h[16 * k + 2 * i], h[16 * k + 2 * i + 1]);
            }
        }
    } else if constexpr (TYPE == kQ3_K) {
        // high-bit mask @0, bit pairs @32, 6-bit scales @96 (per 16 columns), d @108: d * (sc - 32) * ((q2 | hbit << 2) - 4)
        const int n = G >> 2;
        uint32_t hm[8], qs[8];
        words_a2<8>(blk, hm);
        words_a2<8>(blk + 32 + 32 * n, qs);
        const float d = half_bits_to_float(lds16(blk + 108));
        const f32x2 neg_magic = pack2(-(8388608.0f + 4.0f), -(8388608.0f + 4.0f));
#pragma unroll
        for (int k = 0; k < N; ++k) {
            // scales 2 g and 2 g + 1: nibbles of bytes 0..7 (low ones first), two more bits from bytes 8..11, a pair per four scales
            const int g = G + k, j = g & 3;
            const uint32_t sc = ((lds16(blk + 96 + ((2 * g) & 7)) >> (4 * n)) & 0x0F0Fu) | (((lds16(blk + 104 + ((2 * g) & 3)) >> (g & 6)) & 0x0303u) << 4);
            const float dl[2] = {d * static_cast<float>(static_cast<int>(sc & 0xFFu) - 32), d * static_cast<float>(static_cast<int>(sc >> 8) - 32)};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t q = ((qs[i] >> (2 * j)) & 0x03030303u) + ((hm[i] >> g) & 0x01010101u) * 4u;
                bytes_mul_f16(q, neg_magic, pack2(dl[i >> 2], dl[i >> 2]), h[16 * k + 2 * i], h[16 * k + 2 * i + 1]);
            }
        }
    } else if constexpr (TYPE == kQ8_0) {
        // blocks of 32 weights: d @0, 32 int8 @2
        const f32x2 neg_magic = pack2(-(8388608.0f + 128.0f), -(8388608.0f + 128.0f));
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t at = blk + (G + k) * 34;
            const float d = half_bits_to_float(lds16(at));
            uint32_t w[8];
            words_a2<8>(at + 2, w);
#pragma unroll
            for (int i = 0; i < 8; ++i)  // int8 + 128 is the unsigned byte
                bytes_mul_f16(w[i] ^ 0x80808080u, neg_magic, pack2(d, d), h[16 * k + 2 * i], h[16 * k + 2 * i + 1]);
        }
    } else if constexpr (TYPE == kIQ4_XS || TYPE == kIQ4_NL) {
        // byte i of a run of 16: weights i (low nibble) and 16 + i; levels + 128 are looked up four at a time (see iq4_levels4)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int g = G + k;
            uint32_t w[4];
            float dl;
            if constexpr (TYPE == kIQ4_NL) {
                const uint32_t at = blk + g * 18;
                dl = half_bits_to_float(lds16(at));
                words_a2<4>(at + 2, w);
            } else {
                const uint32_t hb = lds16(blk + 2), lb = lds16(blk + 4 + 2 * (g >> 2));  // 6-bit scales: low nibbles @4, high pairs @2
                const uint32_t sc = ((lb >> (4 * (g & 3))) & 15u) | (((hb >> (2 * g)) & 3u) << 4);
                dl = half_bits_to_float(lds16(blk)) * static_cast<float>(static_cast<int>(sc) - 32);
                words_a2<4>(blk + 8 + 16 * g, w);
            }
            const f32x2 neg_magic = pack2(-(8388608.0f + 128.0f), -(8388608.0f + 128.0f)), d2 = pack2(dl, dl);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t a = iq4_levels4(w[i] & 0xFFFFu), b = iq4_levels4(w[i] >> 16);  // nibbles of bytes 0, 1 and 2, 3
                bytes_mul_f16(__byte_perm(a, b, 0x6420), neg_magic, d2, h[16 * k + 2 * i], h[16 * k + 2 * i + 1]);
                bytes_mul_f16(__byte_perm(a, b, 0x7531), neg_magic, d2, h[16 * k + 8 + 2 * i], h[16 * k + 8 + 2 * i + 1]);
            }
        }
    } else {
        constexpr int CPB = chunk_block(TYPE) / 8, BB = chunk_block_bytes(TYPE);
#pragma unroll
        for (int k = 0; k < 4 * N; ++k) {
            const int c = 4 * G + k;
            float v[8];
            deq8<TYPE>(static_cast<const uint8_t *>(__cvta_shared_to_generic(blk + (c / CPB) * BB)), c % CPB, v, table);
#pragma unroll
            for (int e = 0; e < 4; ++e) h[4 * k + e] = f16x2_of(pack2(v[2 * e], v[2 * e + 1]));
        }
    }
}

// ---- the two blocks of a pair ----------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void bar_arrive_cluster(uint32_t cluster_addr) {
    // default semantics, as for a consumer's release of a remote slot; with .release.cluster every slot took 0.2 us longer
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this address in both blocks of pair `pair` once the MMAs issued so far are done
__device__ __forceinline__ void mma_commit_pair(uint32_t bar, uint32_t pair) {
    const uint16_t both = static_cast<uint16_t>(3u << (2 * pair));
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(both)
                 : "memory");
}

struct Tc5Maps {
    CUtensorMap x;     // activations
    CUtensorMap w[8];  // weights, by row class
};

template <int TYPE, int NH>
__global__ void __launch_bounds__(kTThreads, 1) qgemm_tc5_kernel(const __grid_constant__ Tc5Maps maps, const uint8_t *w, float *y, int rows,
                                                                 int cols, long long row_bytes, int ntok, int n_acc, int map_shift, const uint8_t *codebook,
                                                                 unsigned *status) {
    constexpr int CPB = chunk_block(TYPE) / 8, BB = chunk_block_bytes(TYPE);
    constexpr int TABLE = table_bytes16(TYPE);
    constexpr int kTStages = stages_for(TYPE, NH), kXStages = x_stages(NH) < kTStages ? x_stages(NH) : kTStages, kRaw = raw_buffers(TYPE, NH);
    constexpr bool kStaged = raw_staged(TYPE);
    // Decoder warps of a stage, and groups that take turns: a group must not run two uses of a stage ahead of another, the
    // parity of the barriers would not tell them apart, so there are no more groups than stages.
    constexpr int kGroupWarps = kStaged && kTStages >= 4 ? 4 : 8, kGroups = 16 / kGroupWarps;
    static_assert(kGroups <= kTStages, "barrier phases");
    constexpr uint32_t kTmemCols = 256 * NH;
    extern __shared__ uint8_t tc5_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages], s_empty[kMaxStages], s_done, s_raw_full[3], s_raw_empty[3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    // table first, then the stages on a 1024-byte boundary (the swizzle works on absolute shared-memory address bits)
    uint8_t *table = tc5_raw;
    const uint32_t tiles = (s32(tc5_raw) + TABLE + 1023u) & ~1023u;
    constexpr int PITCH = raw_pitch(TYPE), RUN = raw_run_bytes(TYPE);
    const uint32_t x_tiles = tiles + kTStages * kTA, raw_ring = x_tiles + kXStages * (NH * kTB);  // buffers of kTM rows
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // a cluster: `pairs` pairs of blocks that share the columns of 256 weight rows; block `rank` of a pair owns rows rank * 128 ..
    uint32_t cluster_blocks;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cluster_blocks));
    const uint32_t in_cluster = cluster_rank(), rank = in_cluster & 1u;
    const int pairs = static_cast<int>(cluster_blocks >> 1), pair = static_cast<int>(in_cluster >> 1);
    const int row0 = static_cast<int>(blockIdx.x / cluster_blocks) * (2 * kTM) + static_cast<int>(rank) * kTM;
    const int tok0 = blockIdx.y * (NH * n_acc);
    const int n_runs = (cols + kRawCols - 1) / kRawCols;
    const int run0 = pair * n_runs / pairs, run1 = (pair + 1) * n_runs / pairs;  // this pair's columns, in runs of 256
    const int n_k = (run1 * kStagesPerRun < cols / kTK ? run1 * kStagesPerRun : cols / kTK) - run0 * kStagesPerRun;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kTStages; ++s) {
            // one arrive per decoder warp of the group that fills the stage, the feeding thread's with the byte count of the activation tile
            // that goes with it, and in the first block of a pair one more for the second block's stage
            bar_init(s32(&s_full[s]), kGroupWarps + 1 + (rank == 0 ? 1 : 0));
            bar_init(s32(&s_empty[s]), 1);
        }
        bar_init(s32(&s_done), 1);
        for (int b = 0; b < kRaw; ++b) {
            bar_init(s32(&s_raw_full[b]), 1);
            bar_init(s32(&s_raw_empty[b]), kAThreads / 32);  // every decoder warp is done with the buffer
        }
        s_failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (grid_bytes(TYPE) > 0) {
        if constexpr (grid_is_codebook(TYPE)) {
            for (int i = threadIdx.x; i < grid_bytes(TYPE) / 4; i += blockDim.x)
                reinterpret_cast<uint32_t *>(table)[i] = reinterpret_cast<const uint32_t *>(codebook)[i];
        } else {
            if (threadIdx.x < 16) reinterpret_cast<float *>(table)[threadIdx.x] = kIq4Levels[threadIdx.x];
        }
    }
    if (warp == 0) {  // tensor memory: 256 columns per accumulator (one block per SM)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&s_tmem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // the other blocks' barriers and tensor memory exist before anybody signals or multiplies
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    volatile int *failed = &s_failed;

    if (warp < 16) {
        // ---- weight tile: chunk c of the stage (8 weights, 16 bytes of fp16) goes to 16-byte slot c ^ (row % 8) of the row.
        //      "full" is counted per block; the second block of a pair forwards each completed stage to the first block, which
        //      issues the MMAs (such an arrive per producer warp made every half stage take a microsecond).
        const int group = warp / kGroupWarps;
        auto stage_wait = [&](int q) -> bool { return warp_wait(s32(&s_empty[q % kTStages]), ((q / kTStages) & 1) ^ 1, failed); };
        auto stage_done = [&](int q) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            warp_arrive(s32(&s_full[q % kTStages]));
        };
        auto put = [&](int q, int row, int c, uint32_t h0, uint32_t h1, uint32_t h2, uint32_t h3) {
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(tiles + (q % kTStages) * kTA + row * 128 + ((c ^ (row & 7)) << 4)),
                         "r"(h0), "r"(h1), "r"(h2), "r"(h3)
                         : "memory");
        };
        if constexpr (!kStaged) {
            // four threads per row, one chunk each, two rows per thread; rows go 0, 4, 1, 5, ... over a warp's lanes: the 8
            // lanes that the store unit serves together then hit 8 different 16-byte columns of the swizzle
            const int quarter = threadIdx.x & 3, r8 = (threadIdx.x >> 2) & 7;
            const int r = (warp & 7) * 8 + ((r8 >> 1) | ((r8 & 1) << 2));
            const uint8_t *w_row[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) w_row[i] = w + static_cast<size_t>(row0 + r + 64 * i < rows ? row0 + r + 64 * i : 0) * row_bytes;
            for (int q = group; q < n_k; q += kGroups) {
                if (!stage_wait(q)) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = quarter + 4 * (i >> 1), kc = (run0 * kStagesPerRun + q) * (kTK / 8) + c;  // chunk within the stage, the row
                    float v[8];
                    deq8<TYPE>(w_row[i & 1] + static_cast<size_t>(kc / CPB) * BB, kc % CPB, v, table);
                    put(q, r + 64 * (i & 1), c, f16x2_of(pack2(v[0], v[1])), f16x2_of(pack2(v[2], v[3])), f16x2_of(pack2(v[4], v[5])),
                        f16x2_of(pack2(v[6], v[7])));
                }
                stage_done(q);
            }
        } else {
            const int r = (warp & 3) * 32 + lane;
            // position of the row's bytes inside their 16-byte line, and of its class (row % 8) in a buffer
            const uint32_t mis = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(w) + static_cast<size_t>(r & 7) * static_cast<size_t>(row_bytes)) & 15u);
            const int cls = r & 7, slot = (((cls & ((1 << map_shift) - 1)) * 8) >> map_shift) + (cls >> map_shift);
            const uint32_t row_at = raw_ring + (slot * (kTM / 8) + (r >> 3)) * PITCH;
            const int part = kGroups == 4 ? 0 : (warp >> 2) & 1;  // two groups: which 32 columns of a stage
            for (int q = group, run = 0, b = 0, use = 0; q < n_k; q += kGroups) {
                const int in_run = q % kStagesPerRun;
                if (in_run < kGroups && !warp_wait(s32(&s_raw_full[b]), use & 1, failed)) break;  // every lane: it reads the bytes
                const uint32_t blk = row_at + b * (kTM * PITCH) + ((mis + static_cast<uint32_t>(run0 + run) * RUN) & 15u);
                uint32_t h[kGroups == 4 ? 32 : 16];
                decode_slots<TYPE, kGroups == 4 ? 2 : 1>(blk, 2 * in_run + part, table, h);
                if (in_run + kGroups >= kStagesPerRun) {  // the group's last read of the buffer
                    warp_arrive(s32(&s_raw_empty[b]));
                    ++run;
                    if (++b == kRaw) b = 0, ++use;
                }
                if (!stage_wait(q)) break;
#pragma unroll
                for (int c = 0; c < 32 / kGroupWarps; ++c) put(q, r, 4 * part + c, h[4 * c], h[4 * c + 1], h[4 * c + 2], h[4 * c + 3]);
                stage_done(q);
            }
        }
    } else if (warp == 16) {
        // ---- activation tiles: one thread, one TMA tile copy per accumulator and stage (64 columns x half of the
        //      accumulator's activation rows, in the same 128-byte swizzle; no multicast; rows beyond ntok arrive as zeros).
        //      A buffer is refilled once its MMAs are done, which "empty" of their stage says; a tile's bytes are counted on "full" of its
        //      stage.  (With barriers of their own for the activations the MMA warp waited and committed twice per stage.  64 rows of Q4_K
        //      17408 x 5120 40.7 and 39.4 us so, 2048 rows of 5120 x 17408 347 and 341.)
        if (lane == 0) {
            // The kernel is launched while the conversion of the activations may still run (programmatic stream
            // serialization); this thread is the only reader of its output.
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int half = n_acc / 2;
            int k = 0;
            for (; k < n_k; ++k) {
                const int stage = k % kXStages, before = k - kXStages;
                if (before >= 0 && !bar_wait(s32(&s_empty[before % kTStages]), (before / kTStages) & 1, failed)) break;
                const uint32_t bar = s32(&s_full[k % kTStages]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(NH * half * 128) : "memory");
#pragma unroll
                for (int nh = 0; nh < NH; ++nh)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                     x_tiles + stage * (NH * kTB) + nh * kTB),
                                 "l"(&maps.x), "r"(run0 * kRawCols + k * kTK), "r"(tok0 + nh * n_acc + static_cast<int>(rank) * half), "r"(bar)
                                 : "memory");
            }
            // the last tiles land before the block may leave, also when a wait gave up (bounded)
            for (int last = k > kXStages ? k - kXStages : 0; last < k; ++last)
                for (int i = 0; i < (1 << 16) && !bar_try(s32(&s_full[last % kTStages]), (last / kTStages) & 1); ++i) __nanosleep(64);
        }
        __syncwarp();
    } else if (warp == 17) {
        if (rank != 0) {
            // ---- second block of a pair: tell the first block about every stage that is full here
            for (int q = 0; q < n_k; ++q) {
                const int stage = q % kTStages;
                if (!warp_wait(s32(&s_full[stage]), (q / kTStages) & 1, failed)) break;
                if (lane == 0) bar_arrive_cluster(in_block(s32(&s_full[stage]), static_cast<int>(in_cluster & ~1u)));
            }
        } else {
            // ---- MMA issue for both blocks: accumulator nh at column nh * 256.  D fp32, A and B fp16, both K-major, M = 256
            const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(n_acc >> 3) << 17) | ((256u >> 4) << 24);
            for (int q = 0; q < n_k; ++q) {
                const int stage = q % kTStages, xs = q % kXStages;
                if (!__all_sync(0xFFFFFFFFu, bar_wait_cluster(s32(&s_full[stage]), (q / kTStages) & 1, failed) ? 1 : 0)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (tc::elect_one()) {
                    const uint64_t a_desc = sw128_desc(tiles + stage * kTA), b_desc = sw128_desc(x_tiles + xs * (NH * kTB));
#pragma unroll
                    for (int j = 0; j < kTK / 16; ++j)  // 32 bytes further along K inside the swizzled rows per step
#pragma unroll
                        for (int nh = 0; nh < NH; ++nh)
                            mma_f16_pair(tmem + nh * 256, a_desc + 2 * j, b_desc + 2 * j + ((nh * kTB) >> 4), idesc, (q | j) != 0);
                    // the buffers are free again, in both blocks of the pair, once these MMAs have read them
                    mma_commit_pair(s32(&s_empty[stage]), static_cast<uint32_t>(pair));
                }
                __syncwarp();
            }
            if (tc::elect_one()) mma_commit_pair(s32(&s_done), static_cast<uint32_t>(pair));
        }
        __syncwarp();
    } else if constexpr (kStaged) {
        // ---- raw weights: one thread, map c of n brings the rows of classes c, c + n, ... (rows beyond the tensor arrive as zeros)
        if (lane == 0) {
            const int n_maps = 1 << map_shift;
            int issued = 0;
            for (int b = 0, use = 0; issued < run1 - run0; ++issued) {
                if (use > 0 && !bar_wait(s32(&s_raw_empty[b]), (use - 1) & 1, failed)) break;
                const uint32_t bar = s32(&s_raw_full[b]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kTM * PITCH) : "memory");
#pragma unroll 1
                for (int c = 0; c < n_maps; ++c) {
                    const uint32_t mis = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(w) + static_cast<size_t>(c) * static_cast<size_t>(row_bytes)) & 15u);
                    const uint32_t x = ((mis + static_cast<uint32_t>(run0 + issued) * RUN) & ~15u) / kTcElemBytes;
                    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                                     raw_ring + b * (kTM * PITCH) + ((c * 8) >> map_shift) * (kTM / 8) * PITCH),
                                 "l"(&maps.w[c]), "r"(x), "r"(row0 / 8), "r"(0), "r"(bar)
                                 : "memory");
                }
                if (++b == kRaw) b = 0, ++use;
            }
            // the last copies land before the block may leave, also when the decoders gave up (bounded)
            for (int run = issued > kRaw ? issued - kRaw : 0; run < issued; ++run)
                for (int i = 0; i < (1 << 16) && !bar_try(s32(&s_raw_full[run % kRaw]), (run / kRaw) & 1); ++i) __nanosleep(64);
        }
        __syncwarp();
    }

    const int lane_group = warp & 3, col_group = warp >> 2;  // a warp may read the 32 lanes (warp % 4) * 32 onwards
    const uint32_t tm_mine = tmem + (static_cast<uint32_t>(lane_group * 32) << 16);
    const int row = row0 + lane_group * 32 + lane;  // thread = weight row, the warps of a lane group share the column chunks
    bool ok = true;
    if (warp < 16) {
        ok = warp_wait(s32(&s_done), 0, failed);
        // (The next conversion of activations may be launched; it waits for this kernel's end before it touches anything.  Requested at the start
        // of a block, that conversion and the GEMM behind it take SMs that other streams could use: three streams, 1500 rows of Q4_K 17408 x
        // 5120 211 to 243 us, 200 so, 512 rows of four tensors 290 and 284.  One stream alone: 512 rows 80.7 and 80.9, of four tensors 308 and 307.)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    auto read16 = [&](uint32_t at, float (&v)[16]) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
              "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
            : "r"(at)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    };
    auto store16 = [&](int tok, const float (&v)[16]) {
        if (row >= rows) return;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (tok + j < ntok) y[static_cast<size_t>(tok + j) * rows + row] = v[j];
    };
    const int chunks = n_acc / kXChunk;  // of an accumulator
    if (pairs == 1) {
        if (warp < 16 && ok) {
#pragma unroll 1
            for (int c = col_group; c < NH * chunks; c += 4) {
                const int nh = c >= chunks ? 1 : 0, local = c - nh * chunks;
                float v[16];
                read16(tm_mine + nh * 256 + local * kXChunk, v);
                store16(tok0 + nh * n_acc + local * kXChunk, v);
            }
        }
    } else {
#pragma unroll 1
        for (int nh = 0; nh < NH; ++nh) {
            cluster_sync_all();  // everybody's MMAs are done with the stages (and the sums of the round before have been read)
            if (warp < 16) {
#pragma unroll 1
                for (int c = col_group; c < chunks; c += 4) {
                    const int owner = c % pairs;
                    if (owner == pair) continue;
                    float v[16];
                    read16(tm_mine + nh * 256 + c * kXChunk, v);
                    const uint32_t to = in_block(tiles + ((c / pairs) * (pairs - 1) + (pair < owner ? pair : pair - 1)) * kXBytes +
                                                     (lane_group * 32 + lane) * 16,
                                                 owner * 2 + static_cast<int>(rank));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + j * (kTM * 16)), "f"(v[4 * j]), "f"(v[4 * j + 1]),
                                     "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                                     : "memory");
                }
            }
            cluster_sync_all();
            if (warp < 16) {
#pragma unroll 1
                for (int c = pair + pairs * col_group; c < chunks; c += 4 * pairs) {
                    float own[16], v[16];
                    read16(tm_mine + nh * 256 + c * kXChunk, own);
#pragma unroll 1
                    for (int p = 0; p < pairs; ++p) {  // in the order of the columns
                        float from[16];
                        if (p == pair) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) from[j] = own[j];
                        } else {
                            const uint32_t at = tiles + ((c / pairs) * (pairs - 1) + (p < pair ? p : p - 1)) * kXBytes + (lane_group * 32 + lane) * 16;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const uint4 q = lds128u(at + j * (kTM * 16));
                                from[4 * j] = __uint_as_float(q.x), from[4 * j + 1] = __uint_as_float(q.y);
                                from[4 * j + 2] = __uint_as_float(q.z), from[4 * j + 3] = __uint_as_float(q.w);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = p == 0 ? from[j] : v[j] + from[j];
                    }
                    store16(tok0 + nh * n_acc + c * kXChunk, v);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // no block's shared or tensor memory goes away under another
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        if (lane == 0 && s_failed) atomicExch(status, kStatusWaitExpired);
    }
}

// The activations as a 2-D tensor [activation rows][cols] of fp16; a tile is 64 columns (one 128-byte swizzled row each) of
// `box_rows` activation rows, rows beyond the last are zeros.
cudaError_t encode_x_map(CUtensorMap *map, const __half *xh, int cols, int ntok, int box_rows) {
    TcEncode encode = nullptr;
    if (const cudaError_t err = tc_encoder(&encode); err != cudaSuccess) return err;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(ntok)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
    const cuuint32_t box[2] = {kTK, static_cast<cuuint32_t>(box_rows)}, elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(xh), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? cudaSuccess
               : cudaErrorInvalidValue;
}

template <int TYPE, int NH>
struct Tc5Variant {
    static constexpr int kSmem = tc5_smem_bytes(TYPE, NH, stages_for(TYPE, NH));
    static_assert(kSmem <= 227 * 1024, "shared memory of the tcgen05 GEMM");
    static_assert(kSmem - table_bytes16(TYPE) - 1024 >= (kMaxPairs - 1) * (kTNMax / kXChunk / kMaxPairs) * kXBytes, "room for the exchange");
    static constexpr auto kKernel = qgemm_tc5_kernel<TYPE, NH>;

    static void configure(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int row_tiles, int tok_tiles, int pairs, cudaStream_t stream) {
        cfg.gridDim = dim3(static_cast<unsigned>(row_tiles * pairs * 2), static_cast<unsigned>(tok_tiles));
        cfg.blockDim = dim3(kTThreads);
        cfg.dynamicSmemBytes = kSmem;
        cfg.stream = stream;
        // May start while the kernel before it in the stream (the fp32 -> fp16 conversion of the activations) still runs: the
        // set-up, the first weight copies and the first decoded tiles overlap it; the thread that feeds the activations waits.
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = static_cast<unsigned>(pairs * 2);
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
    }
    // clusters of `pairs` pairs that fit on the GPU at once (cached; one device per process), 0 if the kernel cannot run
    static int clusters(int pairs) {
        static int cached[kMaxPairs + 1] = {};
        if (cached[pairs] == 0) {
            int n = 0;
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute attr[2];
            configure(cfg, attr, 1024, 1, pairs, nullptr);
            if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&n, kKernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
            cached[pairs] = n > 0 ? n : -1;
        }
        return cached[pairs] < 0 ? 0 : cached[pairs];
    }
};

// Shape of a launch: accumulators per block (NH), activation rows of each, tiles of activation rows, and how many pairs share
// the columns.  Estimated time in us, fitted to Q6_K 1024 x 5120 and Q4_K 5120 x 17408 with 64 to 512 activation rows, which
// took, alone and in every shape, what this says within 2 us: a wave of clusters walks its share of the stages, pays for start and
// end, and for the sums that the pairs of a cluster send each other.
struct Tc5Plan {
    int nh, n_acc, tok_tiles, pairs;
};
template <int TYPE>
Tc5Plan plan_t(int rows, int cols, int ntok) {
    const int row_tiles = (rows + 2 * kTM - 1) / (2 * kTM), n_runs = (cols + kRawCols - 1) / kRawCols;
    Tc5Plan best{};
    float best_cost = 0.0f;
    for (int nh = 1; nh <= 2; ++nh) {
        const int tok_tiles = (ntok + nh * kTNMax - 1) / (nh * kTNMax);
        const int n_acc = ((ntok + tok_tiles * nh - 1) / (tok_tiles * nh) + 63) / 64 * 64;
        for (int pairs = 1; pairs <= kMaxPairs && pairs <= n_runs; ++pairs) {
            const int fit = nh == 1 ? Tc5Variant<TYPE, 1>::clusters(pairs) : Tc5Variant<TYPE, 2>::clusters(pairs);
            if (fit == 0) continue;
            const int waves = (row_tiles * tok_tiles + fit - 1) / fit, stages = (n_runs + pairs - 1) / pairs * kStagesPerRun;
            const float f = static_cast<float>(n_acc) / 256.0f, both = static_cast<float>(nh) * f;
            const float stage = nh == 1 ? 0.385f + 0.045f * f : 0.44f + 0.16f * f * f;  // decoding bounds one accumulator, the MMAs two
            const float cost = static_cast<float>(waves) * (static_cast<float>(stages) * stage + 9.0f + both +
                                                            (pairs > 1 ? 1.0f + both * (1.6f * static_cast<float>(pairs) - 0.7f) : 0.0f));
            if (best.nh == 0 || cost < best_cost) best = {nh, n_acc, tok_tiles, pairs}, best_cost = cost;
        }
    }
    return best;
}

template <int TYPE>
cudaError_t launch_t(const uint8_t *w, const __half *xh, float *y, int rows, int cols, long long row_bytes, int ntok, const uint8_t *codebook,
                     unsigned *status, cudaStream_t stream) {
    const Tc5Plan plan = plan_t<TYPE>(rows, cols, ntok);
    if (plan.nh == 0) return cudaErrorInvalidConfiguration;
    Tc5Maps maps{};
    cudaError_t err = encode_x_map(&maps.x, xh, cols, ntok, plan.n_acc / 2);
    if (err == cudaSuccess && raw_staged(TYPE)) err = tc_encode_maps(TYPE, w, rows, row_bytes, kTM / 8, maps.w);
    if (err != cudaSuccess) return err;
    const int shift = tc_map_shift(rows, row_bytes);
    const int row_tiles = (rows + 2 * kTM - 1) / (2 * kTM);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    if (plan.nh == 1) {
        Tc5Variant<TYPE, 1>::configure(cfg, attr, row_tiles, plan.tok_tiles, plan.pairs, stream);
        return cudaLaunchKernelEx(&cfg, Tc5Variant<TYPE, 1>::kKernel, maps, w, y, rows, cols, row_bytes, ntok, plan.n_acc, shift, codebook, status);
    }
    Tc5Variant<TYPE, 2>::configure(cfg, attr, row_tiles, plan.tok_tiles, plan.pairs, stream);
    return cudaLaunchKernelEx(&cfg, Tc5Variant<TYPE, 2>::kKernel, maps, w, y, rows, cols, row_bytes, ntok, plan.n_acc, shift, codebook, status);
}

}  // namespace

bool gemm_tc5_supports(int cols) { return cols % kTK == 0; }

cudaError_t launch_qgemm_tc5(int type, const uint8_t *w, const void *xh, float *y, int rows, int cols, long long row_bytes, int ntok,
                             const uint8_t *codebook, unsigned *status, cudaStream_t stream) {
    const __half *x = static_cast<const __half *>(xh);
    switch (type) {
#define VQM_CASE(id, name) \
    case id: return launch_t<id>(w, x, y, rows, cols, row_bytes, ntok, codebook, status, stream);
        VQM_FOR_EACH_TYPE(VQM_CASE)
#undef VQM_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace vqm
