// Batch kNN search with one CTA per query (walk.cuh, frontier_walk.cuh): kernels and launchers, instantiated once per row type
// (search_walk_f32.cu, _f16.cu, _bf16.cu).
//
// Replaces, like search.cu, GetEntryPointsKernel + SearchGraphKernel of the reference
// (cpp/include/cuda_search_kernels.cuh:11-165).
#pragma once
#include <algorithm>

#include "kernels.h"
#include "frontier_walk.cuh"
#include "walk.cuh"

namespace hnsw {

template <class Dist, int W, int P, int kMinCtas>
__global__ void __launch_bounds__(32 * W, kMinCtas) knn_walk_kernel(SearchParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = lane_number();
  Walk<Dist, W, P> walk;
  walk.de.init(make_table(p.g), smem);
  walk.bind(smem + Dist::smem_bytes(p.g.d), p.ef, p.g.stride0, p.vsize, p.g.n);
  walk.rows = p.g.rows0;
  walk.upper_base = p.g.upper_base;
  walk.level = 0;
  walk.self = -1;
  if (threadIdx.x >= 32) {
    walk.help(p.queries);
    return;
  }
  for (;;) {
    long long qi = blockIdx.x;
    if (p.ticket) {
      if (lane == 0) qi = (long long)atomicAdd(p.ticket, 1ull);
      qi = __shfl_sync(FULL, qi, 0);
      if (__any_sync(FULL, qi >= p.nq)) break;
    }
    if (p.order) qi = __ldg(p.order + qi);
    walk.start(kWalkQuery, p.queries, qi);
    int cur;
    float dcur;
    if (p.entry_node) {
      cur = __ldg(p.entry_node + qi);
      dcur = __ldg(p.entry_dist + qi);
    } else {
      walk.descend(p.g, cur, dcur);
    }
    walk.seed(cur, dcur);  // layer 0: list = {entry}, visited = {entry} (cuda_search_kernels.cuh:108-112)
    walk.run();
    // ascending top-k, found = min(size, k); slots past `found` read -1 / +inf
    const int found = min(walk.list.size, p.topk);
    for (int r = lane; r < p.topk; r += 32) {
      int id = -1;
      float dist = __int_as_float(0x7f800000);
      if (r < found) {
        const uint2 k = lds64(walk.list.keys + 8 * r);
        id = (int)(k.y >> 1);
        dist = ord2f(k.x);
        if (p.labels) id = __ldg(p.labels + id);
      }
      p.out_ids[(size_t)qi * p.topk + r] = id;
      p.out_dist[(size_t)qi * p.topk + r] = dist;
    }
    if (lane == 0) p.out_found[qi] = found;
    __syncwarp();
    if (!p.ticket) break;
  }
  walk.finish();
  if (p.stats && lane == 0) {
    atomicAdd(p.stats + 0, (unsigned long long)walk.wc.evals);
    atomicAdd(p.stats + 1, (unsigned long long)walk.wc.expansions);
    atomicAdd(p.stats + 2, (unsigned long long)walk.wc.sweeps);
    atomicAdd(p.stats + 3, (unsigned long long)walk.wc.inserts);
  }
}

// Entries of the visited table: the largest power of two up to `top` that keeps `ctas` CTAs resident per SM, never
// below 4 per list slot (where repeated evaluations explode) unless the table would not fit at all; p.table_request > 0
// is the caller's own figure.  0: does not fit.
template <class Dist, int W, int P>
int walk_table_entries(const SearchParams& p, int ctas, int top) {
  const auto bytes = [&](int v) {
    return (Dist::smem_bytes(p.g.d) + Walk<Dist, W, P>::smem_bytes(p.ef, p.g.stride0, v, p.g.n) + 15) / 16 * 16;
  };
  const auto pow2 = [](long long x) {
    int v = 1;
    while (v < x) v <<= 1;
    return v;
  };
  int v;
  if (p.table_request > 0) {
    v = std::min(32768, std::max(64, pow2(p.table_request)));
  } else {
    const int floor_entries = std::min(4096, std::max(512, pow2(4ll * p.ef)));
    v = top;
    while (v > floor_entries && (bytes(v) + 1024) * ctas > p.smem_per_sm) v >>= 1;
  }
  while (v > 64 && bytes(v) + 2048 > p.smem_optin) v >>= 1;
  return bytes(v) + 2048 > p.smem_optin ? 0 : v;
}

template <class Dist, int W, int P, int kMinCtas>
cudaError_t launch_walk_t(const SearchParams& p0, int table_top, int sm_count, cudaStream_t stream,
                          const SearchSchedule* sched) {
  SearchParams p = p0;
  p.vsize = walk_table_entries<Dist, W, P>(p, kMinCtas, table_top);
  if (p.vsize == 0) return cudaErrorInvalidConfiguration;
  const size_t smem =
      (Dist::smem_bytes(p.g.d) + Walk<Dist, W, P>::smem_bytes(p.ef, p.g.stride0, p.vsize, p.g.n) + 15) / 16 * 16;
  auto kern = knn_walk_kernel<Dist, W, P, kMinCtas>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * W, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const long long grid = std::max(1ll, std::min((long long)per_sm * sm_count, p.nq));
  // more queries than resident walks: start the long ones first
  if (sched && p.nq > grid && p.nq <= sched->capacity && p.nq <= 0x7fffffffll) {
    e = schedule_search(p, *sched, stream);
    if (e != cudaSuccess) return e;
  }
  if (p.nq <= grid) p.ticket = nullptr;  // a CTA for every query: nothing to hand out, and no counter to clear
  else if ((e = cudaMemsetAsync(p.ticket, 0, sizeof(unsigned long long), stream)) != cudaSuccess) return e;
  kern<<<(unsigned)grid, 32 * W, smem, stream>>>(p);
  return cudaGetLastError();
}

// The same on a frontier (frontier_walk.cuh), for few queries.
template <class Dist, int W, int P, int kMinCtas>
__global__ void __launch_bounds__(32 * W, kMinCtas) knn_frontier_kernel(SearchParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = lane_number();
  FrontierWalk<Dist, W, P> walk;
  walk.de.init(make_table(p.g), smem);
  walk.bind(smem + Dist::smem_bytes(p.g.d), p.ef, p.slots, p.g.stride0, p.vsize, p.g.n);
  walk.rows = LayerRows(p.g.rows0, p.g.stride0, p.g.upper_base, 0);
  walk.self = -1;
  if (threadIdx.x >= 32) {
    walk.help(p.queries);
    return;
  }
  for (;;) {
    long long qi = blockIdx.x;
    if (p.ticket) {
      if (lane == 0) qi = (long long)atomicAdd(p.ticket, 1ull);
      qi = __shfl_sync(FULL, qi, 0);
      if (__any_sync(FULL, qi >= p.nq)) break;
    }
    if (p.order) qi = __ldg(p.order + qi);
    walk.start(kWalkQuery, p.queries, qi);
    int cur;
    float dcur;
    if (p.entry_node) {
      cur = __ldg(p.entry_node + qi);
      dcur = __ldg(p.entry_dist + qi);
    } else {
      walk.descend(p.g, cur, dcur);
    }
    walk.seed(cur, dcur);  // layer 0: one key, the entry, which is visited (cuda_search_kernels.cuh:108-112)
    walk.run();
    write_closest(p, qi, walk.fr);
    if (!p.ticket) break;
  }
  walk.finish();
  if (p.stats && lane == 0) {
    atomicAdd(p.stats + 0, (unsigned long long)walk.wc.evals);
    atomicAdd(p.stats + 1, (unsigned long long)walk.wc.expansions);
    atomicAdd(p.stats + 2, (unsigned long long)walk.wc.sweeps);
    atomicAdd(p.stats + 3, (unsigned long long)walk.wc.inserts);
  }
}

// Key slots and visited-table entries: as many entries as keep `ctas` CTAs resident per SM, up to `top`, never
// below four per key (where repeated evaluations explode) unless the table would not fit at all; p.table_request > 0
// is the caller's own figure.  Returns the shared memory of a CTA, 0: does not fit.
template <class Dist, int W, int P>
size_t plan_cta(SearchParams& p, int ctas, int top) {
  const size_t dist = Dist::smem_bytes(p.g.d);
  const auto bytes = [&] { return dist + FrontierWalk<Dist, W, P>::smem_bytes(p.slots, p.g.stride0, p.vsize, p.g.n); };
  p.slots = Frontier::slots_for(p.ef);
  if (p.table_request > 0) {
    p.vsize = 64;
    while (p.vsize < p.table_request && p.vsize < 32768) p.vsize <<= 1;
  } else {
    const int least = std::max(512, std::min(4096, 4 * p.ef)) / 64 * 64;
    p.vsize = std::max(top, least);
    while (p.vsize > least && (bytes() + 1024) * ctas > p.smem_per_sm) p.vsize -= 64;
  }
  if (bytes() + 1024 > p.smem_optin) p.slots = Frontier::least_slots(p.ef);
  while (p.vsize > 64 && bytes() + 1024 > p.smem_optin) p.vsize >>= 1;
  return bytes() + 1024 > p.smem_optin ? 0 : bytes();
}

template <class Dist, int W, int P, int kMinCtas>
cudaError_t launch_frontier_t(const SearchParams& p0, int table_top, int sm_count, cudaStream_t stream,
                              const SearchSchedule* sched) {
  SearchParams p = p0;
  const size_t smem = plan_cta<Dist, W, P>(p, kMinCtas, table_top);
  if (smem == 0) return cudaErrorInvalidConfiguration;
  auto kern = knn_frontier_kernel<Dist, W, P, kMinCtas>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * W, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const long long grid = std::max(1ll, std::min((long long)per_sm * sm_count, p.nq));
  // more queries than resident walks: start the long ones first
  if (sched && p.nq > grid && p.nq <= sched->capacity && p.nq <= 0x7fffffffll) {
    e = schedule_search(p, *sched, stream);
    if (e != cudaSuccess) return e;
  }
  if (p.nq <= grid) p.ticket = nullptr;  // a CTA for every query: nothing to hand out, and no counter to clear
  else if ((e = cudaMemsetAsync(p.ticket, 0, sizeof(unsigned long long), stream)) != cudaSuccess) return e;
  kern<<<(unsigned)grid, 32 * W, smem, stream>>>(p);
  return cudaGetLastError();
}

// Which shape.  Measured (ms per launch on a B200, CUDA tensors; one warp per query / the shape chosen here):
//   1.18 M x 50, ef 200:  1 query 0.264 / 0.142, 148: 0.717 / 0.483, 1000: 1.07 / 0.64, 4000: 1.33 / 1.01,
//                         6000: 1.36 / 1.29 (10 000: 1.46 / 1.99, so not there)
//   500 000 x 128, ef 128: 1: 0.269 / 0.133, 1000: 1.28 / 0.70, 3000: 1.52 / 1.07, 6000: 1.59 / 1.47 (10 000: 1.76 / 2.32)
//   150 000 x 960, ef 300 (the former CTA-per-query kernel / now): 1: 0.338 / 0.251, 300: 1.12 / 0.83, 1000: 1.22 / 1.07
// Short walks prepare four nodes at a time: their later nodes are less certain and their neighbours overlap more (20 000 x
// 50, ef 100: 1.6 evaluations for each distinct row with eight, 1.3 with four).
// Few queries walk on a frontier.  ms, list / frontier, at up to one query per SM, 16 warps x 16 nodes: 148 of 1.18 M x 50, ef 60
// 0.251 / 0.225, ef 200 0.477 / 0.350; 37 of 1 M x 128 whole numbers, ef 64 0.274 / 0.244; 37 of 1 M x 96, ef 64 0.204 / 0.186.  At up to
// three, 8 x 8 in three CTAs per SM: 300 of 300 000 x 96 whole numbers, ef 128 0.443 / 0.369; 300 of 300 000 x 64 f16 0.357 /
// 0.291; 200 of 500 000 x 64 whole numbers 0.483 / 0.416.  At seven it is the data that decides (500 000 x 64 whole numbers, ef 64
// 0.339 / 0.380, ef 256 0.848 / 0.739; 300 000 x 64 f16, ef 60 0.250 / 0.308; 1.18 M x 50, ef 200 0.677 / 0.566).
constexpr int kShortWalk = 100;  // largest ef of a short walk
template <class Dist, int kCtas>
cudaError_t launch_walk_narrow(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  if (p.nq <= sm_count) return launch_frontier_t<Dist, 16, 16, 1>(p, 8192, sm_count, stream, sched);
  if (p.nq <= (long long)sm_count * 3) return launch_frontier_t<Dist, 8, 8, 3>(p, 8192, sm_count, stream, sched);
  if (p.ef <= kShortWalk) return launch_walk_t<Dist, 4, 4, kCtas>(p, 8192, sm_count, stream, sched);
  if (p.nq <= (long long)sm_count * 27) return launch_walk_t<Dist, 4, 8, kCtas>(p, 8192, sm_count, stream, sched);
  return launch_walk_t<Dist, 2, 8, 10>(p, 8192, sm_count, stream, sched);
}
template <class Dist>
cudaError_t launch_walk_wide(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  // on a frontier while the SMs hold all queries at once.  ms, list / frontier: 148 of 150 000 x 960, ef 60 (8 x 4) 0.305 / 0.281;
  // 148 of 300 000 x 300, ef 100 (8 x 8) 0.310 / 0.306; 300 of 150 000 x 960, ef 300 (8 x 8) 0.890 / 0.679; one (16 x 16) 0.326 / 0.253
  if (p.nq <= sm_count) {
    if (p.ef > kShortWalk) return launch_frontier_t<Dist, 16, 16, 1>(p, 16384, sm_count, stream, sched);
    if (p.g.d > 512) return launch_frontier_t<Dist, 8, 4, 2>(p, 16384, sm_count, stream, sched);
  }
  // while two CTAs of eight warps per SM hold all queries at once; further on four CTAs of four serve more (60 000 x 960, 2,
  // 3 and 4 queries per SM, four / eight warps: ef 100 1.21 1.06 0.94, ef 200 1.12 0.96 0.78, ef 400 1.12 0.92 0.73)
  if (p.nq <= (long long)sm_count * 2) return launch_frontier_t<Dist, 8, 8, 2>(p, 16384, sm_count, stream, sched);
  if (p.ef <= kShortWalk) return launch_walk_t<Dist, 4, 4, 4>(p, 16384, sm_count, stream, sched);
  return launch_walk_t<Dist, 4, 8, 4>(p, 16384, sm_count, stream, sched);
}

template <class Row>
cudaError_t launch_search_walk(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  using E = Pick<Row>;
  const int d = p.g.d;
  if (d <= 32) return launch_walk_narrow<typename E::D32, 6>(p, sm_count, stream, sched);
  if (d <= 64) return launch_walk_narrow<typename E::D64, 6>(p, sm_count, stream, sched);
  if (d <= 96) return launch_walk_narrow<typename E::D96, 5>(p, sm_count, stream, sched);
  if (d <= 128) return launch_walk_narrow<typename E::D128, 5>(p, sm_count, stream, sched);
  // a warp gets one to five rows of a round: two rows of eight columns in flight bring a 3840-byte row in one round trip;
  // rows of up to four columns have nothing for the other four to load (300 000 x 300: 0.62 against 0.73 ms)
  if (d <= 512) return launch_walk_wide<typename E::Wide>(p, sm_count, stream, sched);
  return launch_walk_wide<typename E::Team>(p, sm_count, stream, sched);
}

}  // namespace hnsw
