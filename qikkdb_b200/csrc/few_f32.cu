// Aggregation pass of tables that hold every group (groupby_few.cuh), float keys.
#include "groupby_few.cuh"

namespace qdb {
int32_t launch_few_f32(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st) {
    return launch_few_k<float, false>(a, vk, smem, grid, st);
}
}  // namespace qdb
