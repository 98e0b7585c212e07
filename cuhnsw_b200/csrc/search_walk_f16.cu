// One CTA per query over IEEE half rows.
#include "search_walk.cuh"

namespace hnsw {
cudaError_t launch_search_walk_f16(const SearchParams& p, int sm_count, cudaStream_t stream,
                                     const SearchSchedule* sched) {
  return launch_search_walk<RowF16>(p, sm_count, stream, sched);
}
}  // namespace hnsw
