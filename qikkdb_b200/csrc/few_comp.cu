// Aggregation pass of tables that hold every group (groupby_few.cuh), (int32, int32) composite keys.
#include "groupby_few.cuh"

namespace qdb {
int32_t launch_few_comp(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st) {
    return launch_few_k<int32_t, true>(a, vk, smem, grid, st);
}
}  // namespace qdb
