// Host-visible declarations shared by the kernel translation units and the runtime.
#pragma once

#include <cuda.h>  // CUtensorMap (types only; nothing links against the driver)
#include <cuda_runtime.h>

#include <cstdint>

namespace vqm {

constexpr int kMaxParts = 4;  // tensors one launch can cover (they share the activations, the type and the columns)

// Row-sharded matvec across GPUs: where a launch stores its outputs inside every rank's exchange region (plain remote
// stores over NVLink, issued by the lane that holds the output) and which flags order that against the consumers.
struct PushInfo {
    unsigned long long region[8];  // device address of every rank's exchange region, this rank's included
    unsigned *pushes;              // this rank's own count of pushes per slot, unsigned[n_slots] (inside its region)
    long long dst_off[kMaxParts];  // per tensor: byte offset, inside a region, of its gathered y[0][0]
    long long flag_off;            // byte offset, inside a region, of the flag table: unsigned flags[slot][8 ranks], the
                                   // number of pushes of the slot each rank has completed
    int n_ranks, rank;
    int rows_total[kMaxParts];     // per tensor: the gathered tensor has rows_total rows ...
    int row_begin[kMaxParts];      // ... and this rank's slice starts at row_begin
    int push_slot;                 // 1 + flag slot signalled after the push (0: no push)
    int wait_slot;                 // 1 + slot every rank must have pushed as often as this rank before x is read (0: no wait)
};

// One tensor of a launch.  The launch numbers the rows of its tensors consecutively; tensor p owns launch rows
// [row_end of tensor p - 1, row_end).  Unused entries have row_end = INT_MAX.
struct MatvecPart {
    const uint8_t *w;  // raw blocks, readable up to 15 bytes past the end
    float *y;          // [M][rows] fp32 (may be null when only the argmax is wanted)
    int row_end;
    int rows;          // rows of this tensor (the stride of y)
};

struct MatvecArgs {
    MatvecPart part[kMaxParts];
    const float *x;          // [M][cols] fp32, 16-byte aligned
    const uint8_t *codebook;  // device copy of the type's GGUF codebook (IQ2/IQ3 types), else null
    unsigned *status;        // device error word (0 = fine)
    // fused argmax (all null / 0 when unused; single-tensor launches only)
    float *part_val;         // [kMaxTok][gridDim.x]
    int *part_idx;           // [kMaxTok][gridDim.x]
    unsigned *done_counter;  // zero before the launch; the kernel leaves it zero
    int *out_idx;            // [M] winning row (+ row_base), 0x7fffffff if the column has no value above -inf
    float *out_val;          // [M] winning value (may be null)
    int rows, cols;          // rows: of all tensors together
    long long row_bytes;
    int row_base;            // added to row numbers reported by the argmax (row-sharded weights)
    // Column split for short launches: the k_split blocks of a thread-block cluster share a group of rows (one row per
    // warp), each takes a range of the column segments and leaves its partial sums in the shared memory of the
    // cluster's first block, which adds them in the order of k and writes the outputs.
    int k_split;             // chosen by the launcher (from the rows and the columns only, never from M); 1 = off
    int allow_split;         // host only: the caller permits the split
    int overlap_launch;      // host only: launch with programmatic stream serialization (see qmv_kernel)
    int max_grid;            // host only: upper bound on the grid (0 = none); sizes the argmax partial arrays
    // Fused prologue / epilogue (the flags of the reference's megakernel QMV, engine/csrc/common/qwen_mk_abi.h:55-58):
    //   kFuseSiluMul: the activations are silu(x) * x2;  kFuseNorm: then rmsnorm over the columns times norm_w;
    //   kFuseAdd: y += W x instead of y = W x (the outputs already hold the residual).
    int fuse;                // kFuse* bits, 0 = plain matvec
    const float *x2;         // [M][cols], with kFuseSiluMul
    const float *norm_w;     // [cols], with kFuseNorm
    float eps;               // rmsnorm epsilon
    PushInfo push;           // all zero when the tensor is not sharded
};

// What the tensor-core matvec needs beside that; filled in by its launcher, so that no block starts with integer divisions.  (Not
// in MatvecArgs: with these 64 bytes the CUDA-core kernel's small launches take 1 to 3 % longer, 3.07 instead of 2.98 us.)
static_assert(sizeof(MatvecArgs) <= 384, "parameters of the CUDA-core kernel");
struct TcMatvecArgs : MatvecArgs {
    const uint8_t *x_split;  // ready-made B operands of more than 8 activation rows
    float *partials;         // sums of launches whose columns are split, see tc_finish_tile; null: clusters exchange them
    unsigned *partial_counts;  // [tile]: how many column ranges are there; zero before and after a launch
    int tc_groups, tc_split_recip;  // groups of k_split blocks, and 65536 / k_split rounded up
    int tc_steps[9];         // block k of a group takes the 256-column steps [tc_steps[k], tc_steps[k + 1])
    int tc_deal, tc_deal_recip;  // rows of a tile that each block of a cluster finishes, and 65536 / tc_deal rounded up
    int tc_first, tc_end;        // tiles of this launch (a launch may take the last round of another, see choose_tc_tail)
    unsigned char tc_map_shift[kMaxParts];  // log2 of the number of tensor maps of each tensor
};

enum : int { kFuseAdd = 1, kFuseNorm = 2, kFuseSiluMul = 8 };  // (4 is the fused argmax, which has its own fields)

constexpr int kMaxSplit = 8;  // column ranges a row can be split into (the portable cluster size)

enum : unsigned { kStatusOk = 0, kStatusWaitExpired = 1, kStatusPeerWaitExpired = 2 };

// One launcher per GGUF type (vqm_matvec_type.cu).  m: activation rows (1..8); sm_count: SMs of the device;
// grid_out (optional) receives the grid size used.
#define VQM_FOR_EACH_TYPE(X) \
    X(0, F32) X(1, F16) X(8, Q8_0) X(10, Q2_K) X(11, Q3_K) X(12, Q4_K) X(13, Q5_K) X(14, Q6_K) X(16, IQ2_XXS) \
    X(17, IQ2_XS) X(18, IQ3_XXS) X(20, IQ4_NL) X(21, IQ3_S) X(22, IQ2_S) X(23, IQ4_XS)
#define VQM_DECLARE_LAUNCHER(id, name)                                                                            \
    cudaError_t launch_qmv_##name(const MatvecArgs &a, int m, int sm_count, cudaStream_t stream, int *grid_out); \
    cudaError_t launch_qmv_fused_##name(const MatvecArgs &a, int m, int sm_count, cudaStream_t stream, int *grid_out);  // honours a.fuse
VQM_FOR_EACH_TYPE(VQM_DECLARE_LAUNCHER)
#undef VQM_DECLARE_LAUNCHER

constexpr int kTcTileRows = 256;   // rows of a tile of the tensor-core matvec
constexpr int kTcMaxMagnitude = 66;  // of a codebook, for the tensor-core matvec: times 31 it has to fit into the 11 bits of fp16
inline int tc_tiles(const MatvecArgs &a) {
    int n = 0;
    for (int p = 0; p < kMaxParts; ++p) n += (a.part[p].rows + kTcTileRows - 1) / kTcTileRows;
    return n;
}
// Room for the partial sums of a launch whose columns are split.  It holds a record of every block of one that takes each tile at once (not where
// blocks take several tiles): at most sm_count / 2 tiles, sm_count blocks.  The counts, then the records of tc_finish_tile, 2 of a block for up to 8 activation rows, 12 smaller ones for 24.
constexpr bool tc_partials_hold(int n_tiles, int k_split, int sm_count) { return static_cast<long long>(n_tiles) * k_split <= sm_count; }
constexpr size_t tc_partial_count_bytes(int sm_count) { return (static_cast<size_t>(sm_count) * 4 + 255) / 256 * 256; }
constexpr size_t tc_partial_bytes(int sm_count, int m) {
    return tc_partial_count_bytes(sm_count) + static_cast<size_t>(sm_count) * (m <= 8 ? 2 * (4 * kTcTileRows + 32) : 12 * (2 * kTcTileRows + 32)) * 4;
}
constexpr size_t kTcPartialAlign = 256;  // of the room's address; the kernels' accesses to it are of up to 16 bytes
// Size of the scratch for the B operands of more than 8 activation rows that is to hold `need` bytes where `present` do not: a multiple of
// kTcPartialAlign, because room for partial sums lies behind it.  At most 42 KB per 256 columns; 4 MB hold 24576 columns of any type, so that a
// runtime allocates once (with 3.9 MB for partial sums behind them).  (cudaMalloc takes 330 us for any size from 1 to 16 MB; with 2 MB, which
// tensors of more than 12288 columns outgrow, to bind three tensors and their buffers of 24 rows took 1720 us instead of 1480.)  It grows by half
// at least: what it has outgrown, which captured graphs may use, is together at most twice its size.
constexpr size_t tc_grown_split_bytes(size_t need, size_t present) {
    size_t bytes = need < (4u << 20) ? 4u << 20 : need;
    if (bytes < present + present / 2) bytes = present + present / 2;
    return (bytes + kTcPartialAlign - 1) / kTcPartialAlign * kTcPartialAlign;
}
struct TcScratch {
    const uint8_t *x_split = nullptr;  // the B operands of more than 8 activation rows
    // Room for partial sums, aligned to kTcPartialAlign, in use by one launch at a time: counts zero and sums empty (bytes of 0xFF) before and
    // after it.  Null: the blocks that share columns are clusters and exchange sums in shared memory.  The outputs are the same, bit for bit.
    uint8_t *partials = nullptr;
};
// The tensor-core matvec (vqm_tcmv_type.cu).  maps: per tensor of the launch its tensor maps (tc_encode_maps).
#define VQM_FOR_EACH_TC_TYPE(X) \
    X(8, Q8_0) X(10, Q2_K) X(11, Q3_K) X(12, Q4_K) X(13, Q5_K) X(14, Q6_K) X(16, IQ2_XXS) X(17, IQ2_XS) X(18, IQ3_XXS) \
    X(20, IQ4_NL) X(21, IQ3_S) X(22, IQ2_S) X(23, IQ4_XS)
// split_tcmv_*: into how many column ranges the launch would be split (to go into a.k_split), 0 = the CUDA-core kernel is better.
// launch_tcmv_*: n_launched (may be null) is counted up by the kernels launched, one or two (split: one for 16 rows).
#define VQM_DECLARE_TC_LAUNCHER(id, name)                                                                                        \
    int split_tcmv_##name(const MatvecArgs &a, int sm_count);                                                                    \
    cudaError_t launch_tcmv_##name(const MatvecArgs &a, const CUtensorMap *const *maps, int n_parts, const TcScratch &scratch, int m, \
                                   int sm_count, cudaStream_t stream, int *n_launched);
// wide_rows_*: how many activation rows a launch takes, 24, 16 or 8; split_bytes_*: size of x_split for a launch of more than 8 rows over so
// many columns, 0 if the type takes 8 at most; launch_split_*: makes it from a.x.
#define VQM_DECLARE_SPLIT(id, name)                   \
    int wide_rows_##name();                            \
    size_t split_bytes_##name(int cols);               \
    cudaError_t launch_split_##name(const MatvecArgs &a, uint8_t *x_split, int m, cudaStream_t stream, int *n_launched);
VQM_FOR_EACH_TC_TYPE(VQM_DECLARE_SPLIT)
#undef VQM_DECLARE_SPLIT
VQM_FOR_EACH_TC_TYPE(VQM_DECLARE_TC_LAUNCHER)
#undef VQM_DECLARE_TC_LAUNCHER
// box_rows: rows of a class that one copy brings (32: a tile of 256 rows in all)
cudaError_t tc_encode_maps(int type, const uint8_t *w, int rows, long long row_bytes, int box_rows, CUtensorMap *out);

constexpr int kMaxGrid = 4096;  // upper bound on the matvec grid (sizes the argmax partial arrays)

// Prompt-pass GEMM on the tensor cores (vqm_gemm.cu).  xh: fp16 activations [ntok padded to gemm_token_tile()][cols].
int gemm_token_tile();
cudaError_t launch_f32_to_f16_rows(const float *x, void *xh, long long n_valid, long long n_total, cudaStream_t stream);
cudaError_t launch_qgemm(int type, const uint8_t *w, const void *xh, float *y, int rows, int cols, long long row_bytes, int ntok,
                         const uint8_t *codebook, cudaStream_t stream);

// Prompt-pass GEMM on tcgen05 tensor cores with the accumulators in tensor memory (vqm_gemm_tc5.cu); xh: ntok rows, needs
// cols to be a multiple of 64.  status: device word that receives a code if a bounded
// wait expires.
bool gemm_tc5_supports(int cols);
cudaError_t launch_qgemm_tc5(int type, const uint8_t *w, const void *xh, float *y, int rows, int cols, long long row_bytes, int ntok,
                             const uint8_t *codebook, unsigned *status, cudaStream_t stream);

// n16 16-byte words from pinned host memory
cudaError_t launch_fetch(const void *from, void *to, int n16, cudaStream_t stream);
cudaError_t launch_argmax_rows(const float *x, int n, int ntok, int *out, cudaStream_t stream);
cudaError_t launch_dequant(int type, const uint8_t *w, float *out, long long numel, const uint8_t *codebook,
                           cudaStream_t stream);

}  // namespace vqm
