// One translation unit per GGUF type (-DVQM_TYPE=<id> -DVQM_TYPE_NAME=<name>): instantiates the tensor-core matvec for 1, 2,
// up to 4 and up to 8 activation rows and exports its launcher.
#include "vqm_tcmv_kernel.cuh"

#ifndef VQM_TYPE
#error "compile with -DVQM_TYPE=<GGUF type id> -DVQM_TYPE_NAME=<name>"
#endif

namespace vqm {
namespace {

template <int MC, typename MAPS>
struct TcVariant {
    static constexpr int kSmem = tc_smem_bytes<VQM_TYPE, MC>();
    static constexpr auto kKernel = tcmv_kernel<VQM_TYPE, MC, MAPS>;

    // clusters of `k_split` blocks that fit on the GPU at once (cached; one device per process), 0 if the kernel cannot run
    static int clusters(int k_split, int sm_count) {
        static int cached[kMaxSplit + 1] = {};
        if (cached[k_split] != 0) return cached[k_split] < 0 ? 0 : cached[k_split];
        int n = 0;
        cudaError_t err = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (err == cudaSuccess) {
            if (k_split == 1) {
                int per_sm = 0;
                err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kKernel, kTcThreads, kSmem);
                n = per_sm > 0 ? sm_count : 0;  // all of tensor memory is taken: one block per SM
            } else {
                cudaLaunchConfig_t cfg{};
                cudaLaunchAttribute attr[2];
                configure(cfg, attr, k_split * sm_count, k_split, 0, nullptr);
                err = cudaOccupancyMaxActiveClusters(&n, kKernel, &cfg);
            }
        }
        if (err != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
        }
        cached[k_split] = n > 0 ? n : -1;
        return n;
    }

    static void configure(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int grid, int k_split, int overlap, cudaStream_t stream) {
        cfg.gridDim = dim3(static_cast<unsigned>(grid));
        cfg.blockDim = dim3(kTcThreads);
        cfg.dynamicSmemBytes = kSmem;
        cfg.stream = stream;
        int n = 0;
        if (overlap) {
            attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[n].val.programmaticStreamSerializationAllowed = 1;
            ++n;
        }
        if (k_split > 1) {
            attr[n].id = cudaLaunchAttributeClusterDimension;
            attr[n].val.clusterDim.x = static_cast<unsigned>(k_split);
            attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
            ++n;
        }
        cfg.attrs = attr;
        cfg.numAttrs = n;
    }

    static cudaError_t launch(const MatvecArgs &a, const CUtensorMap *const *maps, int n_parts, int n_tiles, int m, int sm_count, cudaStream_t stream) {
        const int fit = clusters(a.k_split, sm_count);
        if (fit == 0) return cudaErrorInvalidConfiguration;
        const int grid = (n_tiles < fit ? n_tiles : fit) * a.k_split;
        MAPS packed;
        for (int p = 0; p < static_cast<int>(sizeof(packed.m) / sizeof(packed.m[0])); ++p)
            for (int c = 0; c < 8; ++c) packed.m[p][c] = maps[p < n_parts ? p : 0][c];
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[2];
        configure(cfg, attr, grid, a.k_split, a.overlap_launch, stream);
        return cudaLaunchKernelEx(&cfg, kKernel, a, packed, m);
    }
};

// Into how many column ranges the rows' sums are split.  Time of a launch in steps of 256 columns: every group of blocks walks
// `rounds` tiles of 256 rows, each block its share of the steps; a tile costs about one step more for its sums (and another
// half for adding them up across a cluster).  Depends on rows and columns only.
inline int choose_tc_split(int n_tiles, int cols, int allow_split, int sm_count) {
    const int n_steps = (cols + kTcStepCols - 1) / kTcStepCols;
    int best = 1;
    float best_cost = 0.0f;
    for (int s = 1; s <= (allow_split ? kMaxSplit : 1) && s <= n_steps; ++s) {
        const int fit = TcVariant<1, TcMaps1>::clusters(s, sm_count);
        if (fit == 0) continue;
        const int groups = n_tiles < fit ? n_tiles : fit, rounds = (n_tiles + groups - 1) / groups;
        const float cost = static_cast<float>(rounds) * (static_cast<float>((n_steps + s - 1) / s) + (s > 1 ? 1.5f : 1.0f));
        if (s == 1 || cost < best_cost) best = s, best_cost = cost;
    }
    return best;
}

}  // namespace

#define VQM_CAT2(a, b) a##b
#define VQM_CAT(a, b) VQM_CAT2(a, b)

cudaError_t VQM_CAT(launch_tcmv_, VQM_TYPE_NAME)(const MatvecArgs &args, const CUtensorMap *const *maps, int n_parts, int m, int sm_count,
                                                 cudaStream_t stream) {
    MatvecArgs a = args;
    int n_tiles = 0;
    for (int p = 0; p < kMaxParts; ++p) n_tiles += (a.part[p].rows + kTcRows - 1) / kTcRows;
    a.k_split = choose_tc_split(n_tiles, a.cols, a.allow_split, sm_count);
    const int n_steps = (a.cols + kTcStepCols - 1) / kTcStepCols;
    for (int k = 0; k <= a.k_split; ++k) a.tc_steps[k] = k * n_steps / a.k_split;
    a.tc_deal = (kTcRows + a.k_split - 1) / a.k_split;
    a.tc_deal_recip = 65536 / a.tc_deal + 1;
    for (int p = 0; p < n_parts; ++p) a.tc_map_shift[p] = static_cast<unsigned char>(tc_map_shift(a.part[p].rows, a.row_bytes));
#define VQM_LAUNCH(MC)                                                                                           \
    (n_parts == 1 ? TcVariant<MC, TcMaps1>::launch(a, maps, n_parts, n_tiles, m, sm_count, stream)                \
                  : TcVariant<MC, TcMaps4>::launch(a, maps, n_parts, n_tiles, m, sm_count, stream))
    if (m == 1) return VQM_LAUNCH(1);
    if (m == 2) return VQM_LAUNCH(2);
    if (m <= 4) return VQM_LAUNCH(4);
    if (m <= 8) return VQM_LAUNCH(8);
    return cudaErrorInvalidValue;
#undef VQM_LAUNCH
}

}  // namespace vqm
