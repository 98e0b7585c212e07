// One CTA per query over bfloat16 rows.
#include "search_walk.cuh"

namespace hnsw {
cudaError_t launch_search_walk_bf16(const SearchParams& p, int sm_count, cudaStream_t stream,
                                      const SearchSchedule* sched) {
  return launch_search_walk<RowBF16>(p, sm_count, stream, sched);
}
}  // namespace hnsw
