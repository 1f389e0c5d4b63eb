// Launchers shared by the GEMM translation units.
#pragma once

#include "gemm_umma.cuh"
#include "gemm_pair_umma.cuh"

#include <atomic>

namespace eider {
namespace gemm {

constexpr uint32_t kPairBlockCode = 512;  // DensePlan::block_n value that selects the CTA-pair kernel
constexpr uint32_t kPairNarrowBlockCode = 384;  // ... and its 256 x 192 form
inline bool is_pair_code(uint32_t block_n) { return block_n == kPairBlockCode || block_n == kPairNarrowBlockCode; }

// Dense GEMMs (row-major output): picks the kernel for the tile code and the kind of output and fills in the column tiles.
// `p.row_tiles` and `p.splits` are set by the caller.
cudaError_t launch_dense(int kind, uint32_t block_n, const CUtensorMap& map_rows, const CUtensorMap& map_cols, Params p, cudaStream_t stream);
// The gate/up GEMM with the SiLU * up -> NVFP4 quantizer in its epilogue.
cudaError_t launch_gated(const CUtensorMap& map_rows, const CUtensorMap& map_cols, Params p, cudaStream_t stream);

namespace {

// Per-device caches: one host process may drive several GPUs, and the shared-memory opt-in, the SM count and the
// cluster occupancy all belong to the device that is current at the call.
constexpr int kMaxDevices = 64;

int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    return dev;
}

int sm_count() {
    static std::atomic<int> count[kMaxDevices];
    const int dev = current_device();
    int c = count[dev].load(std::memory_order_relaxed);
    if (c == 0) {
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
        if (c <= 0) c = 148;
        count[dev].store(c, std::memory_order_relaxed);
    }
    return c;
}

// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device attribute: opt in once on every device that launches.
template <typename Kernel>
cudaError_t opt_in_smem(std::atomic<uint8_t> (&done)[kMaxDevices], Kernel kernel, uint32_t bytes) {
    const int dev = current_device();
    if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t st = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (st == cudaSuccess) done[dev].store(1, std::memory_order_release);
    return st;
}

template <int KIND, int BLOCK_N, bool TRANSPOSED, int TERMS, bool GROUPED, int EPI_WARPS = 4, bool ANY_OUTPUT = false>
cudaError_t launch(const CUtensorMap& map_rows, const CUtensorMap& map_cols, const Params& p, uint32_t work_items,
                   cudaStream_t stream, const ShortRows<GROUPED>& short_rows = {}) {
    constexpr int kStages = default_stages<KIND, BLOCK_N>();
    constexpr uint32_t kSmem = smem_bytes<KIND, BLOCK_N, kStages>();
    auto kernel = gemm_kernel<KIND, BLOCK_N, kStages, TRANSPOSED, TERMS, GROUPED, EPI_WARPS, ANY_OUTPUT>;
    static std::atomic<uint8_t> configured[kMaxDevices];
    if (cudaError_t st = opt_in_smem(configured, kernel, kSmem); st != cudaSuccess) return st;
    uint32_t grid = static_cast<uint32_t>(sm_count());
    if (work_items < grid) grid = work_items;
    if (grid == 0) return cudaSuccess;
    // Programmatic dependent launch: this kernel's prologue (barriers, tensor memory, first weight tiles) may overlap the
    // tail of the kernel before it; everything that kernel wrote is read only after griddepcontrol.wait.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(64 + 32 * EPI_WARPS);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, map_rows, map_cols, p, short_rows);
}

// CTA-pair kernel: clusters of two along x, as many pairs as can be co-resident (one CTA per SM).
template <int KIND, uint32_t PAIR_N, bool GATED, bool ANY_OUTPUT>
cudaError_t launch_pair(const CUtensorMap& map_rows, const CUtensorMap& map_cols, const Params& p, uint32_t pair_items,
                        cudaStream_t stream) {
    using L = PairSmem<KIND, PAIR_N>;
    auto kernel = gemm_pair_kernel<KIND, PAIR_N, GATED, ANY_OUTPUT>;
    static std::atomic<int> max_pairs_of[kMaxDevices];
    const int dev = current_device();
    int max_pairs = max_pairs_of[dev].load(std::memory_order_acquire);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GATED ? 64 + 32 * kGatedEpilogueWarps : kNumThreads);
    cfg.dynamicSmemBytes = L::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    if (max_pairs == 0) {
        cudaError_t st = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(L::kBytes));
        if (st != cudaSuccess) return st;
        cfg.gridDim = dim3(static_cast<uint32_t>(sm_count()) & ~1u);
        cfg.numAttrs = 1;
        int clusters = 0;
        st = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (st != cudaSuccess) return st;
        if (clusters <= 0) return cudaErrorLaunchOutOfResources;
        max_pairs = clusters;
        max_pairs_of[dev].store(clusters, std::memory_order_release);
    }
    uint32_t grid_pairs = static_cast<uint32_t>(max_pairs);
    if (pair_items < grid_pairs) grid_pairs = pair_items;
    if (grid_pairs == 0) return cudaSuccess;
    cfg.gridDim = dim3(grid_pairs * 2);
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, map_rows, map_cols, p);
}

}  // namespace
}  // namespace gemm
}  // namespace eider
