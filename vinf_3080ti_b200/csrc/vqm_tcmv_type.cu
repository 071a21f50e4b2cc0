// One translation unit per GGUF type (-DVQM_TYPE=<id> -DVQM_TYPE_NAME=<name>): instantiates the tensor-core matvec for 1, 2,
// up to 4, up to 8 and (most types) up to 16 and 24 activation rows and exports its launcher.
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

    // cluster: blocks of a cluster
    static void configure(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int grid, int cluster, int overlap, cudaStream_t stream) {
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
        if (cluster > 1) {
            attr[n].id = cudaLaunchAttributeClusterDimension;
            attr[n].val.clusterDim.x = static_cast<unsigned>(cluster);
            attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
            ++n;
        }
        cfg.attrs = attr;
        cfg.numAttrs = n;
    }

    static cudaError_t launch(TcMatvecArgs &a, const CUtensorMap *const *maps, int n_parts, int n_tiles, int m, int sm_count, cudaStream_t stream) {
        const bool clustered = a.k_split > 1 && a.partials == nullptr;
        const int fit = clustered ? clusters(a.k_split, sm_count) : clusters(1, sm_count) / a.k_split;
        if (fit == 0) return cudaErrorInvalidConfiguration;
        a.tc_groups = n_tiles < fit ? n_tiles : fit;
        a.tc_split_recip = 65536 / a.k_split + 1;
        MAPS packed;
        for (int p = 0; p < static_cast<int>(sizeof(packed.m) / sizeof(packed.m[0])); ++p)
            for (int c = 0; c < 8; ++c) packed.m[p][c] = maps[p < n_parts ? p : 0][c];
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[2];
        configure(cfg, attr, a.tc_groups * a.k_split, clustered ? a.k_split : 1, a.overlap_launch, stream);
        return cudaLaunchKernelEx(&cfg, kKernel, a, packed, m);
    }
};

// Tall tensors, whose blocks walk whole rows: the last round of tiles may occupy a few SMs only (LM head, 151936 rows: 594 tiles
// on 148 SMs, 2 of them in a fifth round).  Its tiles then go to a second launch that splits their columns, if that saves more
// than a launch costs (3.4 us, two to three steps); that launch's blocks are clusters.  first: its first tile, 0 if there is none.
struct TcTail {
    int first = 0, k_split = 0;
};
inline TcTail choose_tc_tail(int n_tiles, int cols, int sm_count, int k_split) {
    const int n_steps = (cols + kTcStepCols - 1) / kTcStepCols, fit1 = TcVariant<1, TcMaps1>::clusters(1, sm_count);
    if (k_split != 1 || fit1 == 0 || n_tiles <= fit1 || n_tiles % fit1 == 0) return {};
    const int rest = n_tiles % fit1;
    int best = 0, best_steps = n_steps;
    for (int s = 2; s <= kMaxSplit && s <= n_steps; ++s)
        if (rest <= TcVariant<1, TcMaps1>::clusters(s, sm_count) && (n_steps + s - 1) / s < best_steps) best = s, best_steps = (n_steps + s - 1) / s;
    if (best == 0 || best_steps + 4 > n_steps) return {};
    return {n_tiles - rest, best};
}

// (one tensor; an argmax is merged through its values)
inline bool takes_tail(const MatvecArgs &a) { return a.part[1].rows == 0 && (a.out_idx == nullptr || a.out_val != nullptr); }

// Into how many column ranges the rows' sums are split, 0 if the launch is too small for this kernel.  Depends on rows and
// columns only.
// Time of a launch in steps of 256 columns: every group of blocks walks `rounds` tiles of 256 rows, each block its share of the
// steps (pairs of warp groups take whole steps in turn: an odd number costs as much as the next even one); a tile costs about
// one step more for its sums, and another half for adding them up across blocks.  As many groups run at once as clusters find room, also
// where the sums go through memory, which needs none: a launch has to give the same bits either way, so it has the same split.
// A launch has a fixed cost of about 3.4 us here and of 2.6 us on the CUDA-core kernel, which reads all columns of a short
// tensor at once while a block here walks its steps; but it takes a quarter of the SMs, and more rows cost it little.  So
// where the line lies depends on what else the GPU does.  Measured with 1 / 4 / 8 rows, CUDA-core and this one (us):
//   launches that wait for one another, on one stream:
//     Q4_K 1024 x 5120:   5.0 /  6.9 / 10.0  and   6.6 /  7.3 /  9.3      2048 x 5120:  6.6 / 10.3 / 16.2  and   6.7 /  7.4 /  9.5
//     Q6_K 1024 x 5120:   5.3 /  7.5 / 11.1  and   8.6 /  8.9 / 10.1      2048 x 5120:  7.0 / 10.8 / 16.4  and   8.9 /  9.2 / 10.4
//     Q3_K 1024 x 5120:   5.2 /  7.4 / 11.1  and   7.3 /  8.2 /  9.8      2048 x 5120:  6.9 / 10.5 / 16.1  and   7.4 /  8.3 /  9.8
//     IQ3_S 1024 x 5120:  6.8 / 11.2 / 16.9  and   9.7 / 10.2 / 12.1      2048 x 5120:  9.8 / 17.8 / 29.1  and   9.8 / 10.4 / 12.2
//     IQ4_XS 1024 x 5120: 5.3 /  7.0 / 10.0  and   8.1 / 10.5 / 13.3      2048 x 5120:  7.3 / 10.1 / 15.5  and   8.2 / 10.7 / 13.5
//   three runtimes in turn, each on its stream (about 3 is the call itself):
//     Q6_K 1024 x 5120:   4.8 /  6.1 /  8.7  and   3.5 /  3.7 /  4.2      2048 x 5120:  5.8 /  8.5 / 12.6  and   3.7 /  4.0 /  4.4
//     IQ4_XS 1024 x 5120: 4.8 /  6.1 /  8.3  and   3.4 /  4.1 /  5.2      2048 x 5120:  6.1 /  8.3 / 12.9  and   3.6 /  4.3 /  5.4
//   a decoder layer of the 27B model whose 1024 x 5120 projections run there or here (the blocks of the one kernel fit beside nothing of the
//   other), 1 row, 4 with prologues, 8 in groups:  one stream, one graph: 80 / 113 / 86 and 86 / 104 / 85;  three streams: 66 / 94 / 70 and
//   58 / 73 / 69
// The choice must not depend on the number of rows.  From 72 pieces of 256 x 256 weights on, of which no block has to walk more
// than one in 20, launches go here: single rows on one stream pay up to 1.6 times for the shortest of them (8 % of a layer),
// 4 rows and whatever shares the GPU gain more.
inline int choose_tc_split(int n_tiles, int cols, int sm_count, bool single) {
    const int n_steps = (cols + kTcStepCols - 1) / kTcStepCols;
    if (static_cast<long long>(n_tiles) * n_steps < 72) return 0;
    int best = 0, best_walk = 0;
    float best_cost = 0.0f;
    for (int s = 1; s <= kMaxSplit && s <= n_steps; ++s) {
        const int fit = TcVariant<1, TcMaps1>::clusters(s, sm_count);
        if (fit == 0) continue;
        const int groups = n_tiles < fit ? n_tiles : fit, rounds = (n_tiles + groups - 1) / groups, steps = (n_steps + s - 1) / s;
        const int walk = tc_wide(VQM_TYPE) ? (rounds * steps + 1) / 2 * 2 : rounds * steps;
        float cost = static_cast<float>(walk) + static_cast<float>(rounds) * (s > 1 ? 1.5f : 1.0f);
        int walked = rounds * steps;
        if (const TcTail tail = s == 1 ? choose_tc_tail(n_tiles, cols, sm_count, s) : TcTail{}; single && tail.first > 0) {
            walked = (rounds - 1) * steps + (steps + tail.k_split - 1) / tail.k_split;
            cost = static_cast<float>(walked + rounds) + 3.0f;
        }
        if (best == 0 || cost < best_cost) best = s, best_cost = cost, best_walk = walked;
    }
    return static_cast<long long>(n_tiles) * n_steps >= 20ll * best_walk ? best : 0;
}

// More than 8 activation rows (templates, so that types without the variant do not compile it)
template <int TYPE>
constexpr int wide_rows() { return tc_twenty_four<TYPE>() ? 24 : tc_sixteen(TYPE) ? 16 : 8; }
template <int TYPE, int MC>
cudaError_t launch_wide(TcMatvecArgs &a, const CUtensorMap *const *maps, int n_tiles, int m, int sm_count, cudaStream_t stream) {
    if constexpr (MC <= wide_rows<TYPE>()) {
        if (a.x_split == nullptr || a.fuse != 0 || a.out_idx != nullptr) return cudaErrorInvalidValue;
        return TcVariant<(TYPE >= 0 ? MC : 0), TcMaps1>::launch(a, maps, 1, n_tiles, m, sm_count, stream);
    } else {
        return cudaErrorInvalidValue;
    }
}
template <int TYPE, int MC>
cudaError_t split_wide(const MatvecArgs &a, uint8_t *x_split, int m, cudaStream_t stream, int *n_launched) {
    if constexpr (MC <= wide_rows<TYPE>()) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[1];
        cfg.gridDim = dim3(static_cast<unsigned>((a.cols + kTcStepCols - 1) / kTcStepCols));
        cfg.blockDim = dim3(16 * 32);
        cfg.stream = stream;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = a.overlap_launch ? 1 : 0;
        cudaError_t err = cudaSuccess;
        for (int t0 = 0; t0 < m && err == cudaSuccess; t0 += 16) {
            if (n_launched != nullptr) ++*n_launched;
            err = cudaLaunchKernelEx(&cfg, tc_split_kernel<TYPE, MC>, a, x_split, t0, m);
        }
        return err;
    } else {
        return cudaErrorInvalidValue;
    }
}

// Tiles [first, end) of a launch.
inline cudaError_t launch_tiles(const MatvecArgs &args, const CUtensorMap *const *maps, int n_parts, const TcScratch &scratch, int first, int end, int m,
                                int sm_count, cudaStream_t stream, int *n_launched) {
    TcMatvecArgs a{args};
    a.x_split = scratch.x_split;
    if (scratch.partials != nullptr && a.k_split > 1) {
        if (reinterpret_cast<uintptr_t>(scratch.partials) % kTcPartialAlign != 0 || !tc_partials_hold(end - first, a.k_split, sm_count)) return cudaErrorInvalidValue;
        a.partial_counts = reinterpret_cast<unsigned *>(scratch.partials);
        a.partials = reinterpret_cast<float *>(scratch.partials + tc_partial_count_bytes(sm_count));
    }
    const int n_steps = (a.cols + kTcStepCols - 1) / kTcStepCols;
    for (int k = 0; k <= a.k_split; ++k) a.tc_steps[k] = k * n_steps / a.k_split;
    a.tc_deal = (kTcRows + a.k_split - 1) / a.k_split;
    a.tc_deal_recip = 65536 / a.tc_deal + 1;
    a.tc_first = first, a.tc_end = end;
    for (int p = 0; p < n_parts; ++p) a.tc_map_shift[p] = static_cast<unsigned char>(tc_map_shift(a.part[p].rows, a.row_bytes));
    if (n_launched != nullptr) ++*n_launched;
#define VQM_LAUNCH(MC)                                                                                                  \
    (n_parts == 1 ? TcVariant<MC, TcMaps1>::launch(a, maps, n_parts, end - first, m, sm_count, stream)                \
                  : TcVariant<MC, TcMaps4>::launch(a, maps, n_parts, end - first, m, sm_count, stream))
    if (m == 1) return VQM_LAUNCH(1);
    if (m == 2) return VQM_LAUNCH(2);
    if (m <= 4) return VQM_LAUNCH(4);
    if (m <= 8) return VQM_LAUNCH(8);
    if (m <= 16 && n_parts == 1) return launch_wide<VQM_TYPE, 16>(a, maps, end - first, m, sm_count, stream);
    if (m <= 24 && n_parts == 1) return launch_wide<VQM_TYPE, 24>(a, maps, end - first, m, sm_count, stream);
    return cudaErrorInvalidValue;
#undef VQM_LAUNCH
}

}  // namespace

#define VQM_CAT2(a, b) a##b
#define VQM_CAT(a, b) VQM_CAT2(a, b)

int VQM_CAT(split_tcmv_, VQM_TYPE_NAME)(const MatvecArgs &a, int sm_count) {
    return choose_tc_split(tc_tiles(a), a.cols, sm_count, takes_tail(a));
}

int VQM_CAT(wide_rows_, VQM_TYPE_NAME)() { return wide_rows<VQM_TYPE>(); }

size_t VQM_CAT(split_bytes_, VQM_TYPE_NAME)(int cols) {
    constexpr int kRows = wide_rows<VQM_TYPE>();
    return kRows > 8 ? static_cast<size_t>((cols + kTcStepCols - 1) / kTcStepCols) * tc_split_bytes<VQM_TYPE, kRows>() : 0;
}

cudaError_t VQM_CAT(launch_split_, VQM_TYPE_NAME)(const MatvecArgs &a, uint8_t *x_split, int m, cudaStream_t stream, int *n_launched) {
    return m <= 16 ? split_wide<VQM_TYPE, 16>(a, x_split, m, stream, n_launched) : split_wide<VQM_TYPE, 24>(a, x_split, m, stream, n_launched);
}

cudaError_t VQM_CAT(launch_tcmv_, VQM_TYPE_NAME)(const MatvecArgs &args, const CUtensorMap *const *maps, int n_parts, const TcScratch &scratch, int m,
                                                 int sm_count, cudaStream_t stream, int *n_launched) {
    const int n_tiles = tc_tiles(args);
    const TcTail tail = takes_tail(args) ? choose_tc_tail(n_tiles, args.cols, sm_count, args.k_split) : TcTail{};
    if (tail.first == 0) return launch_tiles(args, maps, n_parts, scratch, 0, n_tiles, m, sm_count, stream, n_launched);
    // the whole rounds, then the rest
    const cudaError_t err = launch_tiles(args, maps, n_parts, scratch, 0, tail.first, m, sm_count, stream, n_launched);
    if (err != cudaSuccess) return err;
    MatvecArgs a = args;
    a.k_split = tail.k_split;
    return launch_tiles(a, maps, n_parts, scratch, tail.first, n_tiles, m, sm_count, stream, n_launched);
}

}  // namespace vqm
