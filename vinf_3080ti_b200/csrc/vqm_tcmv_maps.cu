// Host side of the TMA tile copies: the driver's encoder, and the tensor maps of a weight tensor.
#include "vqm_tcmv.cuh"

namespace vqm {

cudaError_t tc_encoder(TcEncode *out) {
    static TcEncode encode = nullptr;
    if (encode == nullptr) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
        if (err != cudaSuccess) return err;
        if (fn == nullptr || found != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        encode = reinterpret_cast<TcEncode>(fn);
    }
    *out = encode;
    return cudaSuccess;
}

// The rows as a three-dimensional array: bytes of a row, row / 8 (stride 8 * row_bytes), row % 8 - the row class - (stride
// row_bytes).  A map's base and strides have to be multiples of 16 bytes, so classes share a map where the row stride allows
// it: classes c, c + n, c + 2n, ... with n * row_bytes a multiple of 16 (n = 1, 2, 4 or 8 maps).  The base is row c's address
// rounded down to 16; the kernel rounds its x coordinates down to 16 bytes and finds the row's first byte behind the
// remainder.  A copy never reads past the tensor: with a number of rows that is no multiple of 8 every class has a map of its
// own, with its own number of rows.
// (Eight copies per stage instead of one cost 1.2 us at a launch's start: each map is fetched on its own.)
cudaError_t tc_encode_maps(int type, const uint8_t *w, int rows, long long row_bytes, int box_rows, CUtensorMap *out) {
    TcEncode encode = nullptr;
    if (const cudaError_t err = tc_encoder(&encode); err != cudaSuccess) return err;
    const cuuint32_t elem = kTcElemBytes;
    const int n = 1 << tc_map_shift(rows, row_bytes);
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(tc_pitch(type)) / elem, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(8 / n)}, step[3] = {1, 1, 1};
    const cuuint64_t stride[2] = {static_cast<cuuint64_t>(row_bytes) * 8, static_cast<cuuint64_t>(row_bytes) * (n == 8 ? 8 : n)};
    for (int c = 0; c < n; ++c) {
        const int first = c < rows ? c : 0;  // (a class without rows is copied from somewhere valid and never used)
        const uintptr_t at = reinterpret_cast<uintptr_t>(w) + static_cast<uintptr_t>(first) * static_cast<uintptr_t>(row_bytes);
        const cuuint64_t dims[3] = {(static_cast<cuuint64_t>(row_bytes) + (at & 15u)) / elem, static_cast<cuuint64_t>((rows - first + 7) / 8),
                                    static_cast<cuuint64_t>(8 / n)};
        if (encode(out + c, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, reinterpret_cast<void *>(at & ~static_cast<uintptr_t>(15)), dims, stride, box, step,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

}  // namespace vqm
