// Aggregation pass of tables that hold every group (groupby_few.cuh), int64_t keys.
#include "groupby_few.cuh"

namespace qdb {
int32_t launch_few_i64(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st) {
    return launch_few_k<int64_t, false>(a, vk, smem, grid, st);
}
}  // namespace qdb
