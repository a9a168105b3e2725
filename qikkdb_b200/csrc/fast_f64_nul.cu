// Fast aggregation pass of calls with NULL masks or a row mask, double keys (groupby_fast.cuh).
#include "groupby_fast.cuh"

namespace qdb {
int32_t launch_fast_f64_nul(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st) {
    return launch_fast_nul_k<double>(a, vk, smem, st);
}
}  // namespace qdb
