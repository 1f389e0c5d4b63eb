// The dense GEMM kernels (row-major output), apart from the decode and grouped forms so that both compile side by side.
#include "gemm_launch.cuh"

namespace eider {
namespace gemm {
namespace {

template <int KIND, bool ANY_OUTPUT>
cudaError_t dispatch(uint32_t block_n, const CUtensorMap& map_rows, const CUtensorMap& map_cols, Params& p, cudaStream_t stream) {
    const uint32_t tile_n = block_n == kPairBlockCode ? kPairN : block_n == kPairNarrowBlockCode ? kPairNarrowN : block_n;
    p.col_tiles = (p.cols + tile_n - 1) / tile_n;
    const uint32_t pair_items = ((p.row_tiles + 1) / 2) * p.col_tiles * p.splits;
    const uint32_t items = p.row_tiles * p.col_tiles * p.splits;
    switch (block_n) {
        case kPairBlockCode: return launch_pair<KIND, kPairN, false, ANY_OUTPUT>(map_rows, map_cols, p, pair_items, stream);
        case kPairNarrowBlockCode: return launch_pair<KIND, kPairNarrowN, false, ANY_OUTPUT>(map_rows, map_cols, p, pair_items, stream);
        case 256: return launch<KIND, 256, false, 1, false, 4, ANY_OUTPUT>(map_rows, map_cols, p, items, stream);
        case 192: return launch<KIND, 192, false, 1, false, 4, ANY_OUTPUT>(map_rows, map_cols, p, items, stream);
        case 128: return launch<KIND, 128, false, 1, false, 4, ANY_OUTPUT>(map_rows, map_cols, p, items, stream);
        default: return launch<KIND, 64, false, 1, false, 4, ANY_OUTPUT>(map_rows, map_cols, p, items, stream);
    }
}

}  // namespace

cudaError_t launch_dense(int kind, uint32_t block_n, const CUtensorMap& map_rows, const CUtensorMap& map_cols, Params p, cudaStream_t stream) {
    const bool plain = epilogue_kind(p) == kEpiBf16;
    if (kind == kNvf4)
        return plain ? dispatch<kNvf4, false>(block_n, map_rows, map_cols, p, stream) : dispatch<kNvf4, true>(block_n, map_rows, map_cols, p, stream);
    return plain ? dispatch<kFp8, false>(block_n, map_rows, map_cols, p, stream) : dispatch<kFp8, true>(block_n, map_rows, map_cols, p, stream);
}

cudaError_t launch_gated(const CUtensorMap& map_rows, const CUtensorMap& map_cols, Params p, cudaStream_t stream) {
    p.col_tiles = p.gate_rows / kGatedFeatures;
    return launch_pair<kNvf4, kPairN, true, false>(map_rows, map_cols, p, ((p.row_tiles + 1) / 2) * p.col_tiles, stream);
}

}  // namespace gemm
}  // namespace eider
