// Aggregation pass of tables that hold every group (groupby_few.cuh), int32_t keys.
#include "groupby_few.cuh"

namespace qdb {
int32_t launch_few_i32(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st) {
    return launch_few_k<int32_t, false>(a, vk, smem, grid, st);
}
}  // namespace qdb
