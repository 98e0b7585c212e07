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
    walk.start(p.queries, qi);
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

// The same on a frontier (frontier_walk.cuh), for few queries and long walks.
template <class Dist, int W, int P, int kMinCtas>
__global__ void __launch_bounds__(32 * W, kMinCtas) knn_frontier_kernel(SearchParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = lane_number();
  FrontierWalk<Dist, W, P> walk;
  walk.de.init(make_table(p.g), smem);
  walk.bind(smem + Dist::smem_bytes(p.g.d), p.ef, p.slots, p.g.stride0, p.vsize, p.g.n);
  walk.rows = LayerRows(p.g.rows0, p.g.stride0, p.g.upper_base, 0);
  walk.self = -1;
  using Board = typename FrontierWalk<Dist, W, P>::Board;
  constexpr bool kShared = W > 4;  // write_ranked
  if (threadIdx.x >= 32) {
    if constexpr (kShared) {
      while (walk.help(p.queries) != kWalkOver) {
        write_ranked(p, (unsigned)walk.posted(Board::kQuery), walk.fr, walk.posted(Board::kPool), walk.warp(), W);
        __syncthreads();
      }
    } else {
      walk.help(p.queries);
    }
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
    if (!kShared || p.topk <= 32) {
      write_closest(p, qi, walk.fr);
    } else {
      if (lane == 0) sts32(walk.board + Board::kPool, walk.fr.done);
      walk.post(kWalkKeys);
      write_ranked(p, qi, walk.fr, walk.fr.done, 0, W);
      __syncthreads();
    }
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

// Short walks prepare four nodes at a time: their later nodes are less certain and their neighbours overlap more (20 000 x
// 50, ef 100: 1.6 evaluations for each distinct row with eight, 1.3 with four).
//
// List or frontier, ms of device time with the L2 cache emptied before each launch.  Up to one query per SM 16 warps x 16 nodes: one of 100 000 x 50, ef 300 0.261 / 0.181; 148 of 1.18 M x 50,
// ef 60 0.251 / 0.225, ef 200 0.477 / 0.350; 37 of 1 M x 128 whole numbers, ef 64 0.274 / 0.244; one and 148 of 600 000 x 50, ef 1500 1.27 /
// 0.72 and 3.01 / 1.60; but ef 10 0.049 / 0.055 and 0.080 / 0.092, ef 25 the same.  Up to three 8 x 8 in three CTAs per SM: 300 of 300 000 x
// 96 whole numbers, ef 128 0.443 / 0.369; 300 of 300 000 x 64 f16 0.357 / 0.291.
// Beyond, short and middling walks are faster on the one or on the other by the data (1000 of 500 000 x 64 whole numbers, ef 64
// 0.339 / 0.408, ef 128 0.485 / 0.529; of 300 000 x 96 0.400 / 0.394, 0.540 / 0.499) and get the list, long ones are not slower on the
// frontier on any of nine tables: 600, 1000 and 2000 of 1.18 M x 50, ef 200 0.67 / 0.55, 0.67 / 0.61, 0.76 / 0.66, ef 400 1.19 / 0.89; of
// 300 000 x 64 f16 0.43 / 0.36, 0.49 / 0.42, 0.58 / 0.56, ef 400 0.95 / 0.83; of 1 M x 128 whole numbers 0.84 / 0.83, 0.95 / 0.95, 1.12 / 1.08, 1.92 /
// 1.94 (4000: 1.95 / 2.20); 1000 of 50 000 x 40, ef 700 1.20 / 0.80; rows of up to 32 values 0.515 / 0.595 at 2000, ef 200.
constexpr int kShortWalk = 100;      // largest ef of a short walk
// Smallest ef on a frontier: of a handful of queries, of up to one per SM and more, of more than one per SM of fp32 rows above 64
// values, whose evaluations a list's other warps share as well, and of up to two per SM of rows above 128 values (of 513 and more: from
// kShortWalk on).  A frontier saves the merges and costs more per neighbour, so it gains the less the warmer the caches.  Time on the list over
// that on the frontier, vectors and links in the L2 cache (a program that asks again and again) / not, at ef 48, 58, 80, 100:
//   one query:  100 000 x 50 0.94 0.97 1.03 1.07; 1.18 M x 50 0.93 0.95 1.03 1.09 / - 1.09 1.14 1.13; 60 000 x 90 f16, 48 links, 0.94 0.98 1.07 1.16;
//               150 000 x 120 0.91 0.91 0.98 1.05 / 0.95 0.98 1.05 1.09; 50 000 x 24 0.93 0.97 1.04 1.10
//   37:         0.96 1.00 1.06 1.11; 1.00 1.05 1.14 1.17; 0.94 0.98 1.05 1.15; 0.99 1.03 1.11 1.14; 0.96 0.98 1.04 1.10
//   148:        0.98 1.00 1.07 1.11; 1.02 1.06 1.13 1.19 / 1.04 1.10 1.11 1.15; 0.97 0.99 1.05 1.13; 0.96 0.98 1.05 1.12 / 1.02 1.05 1.11 1.13; 0.94 0.98 1.03 1.08
//   444:        0.97 0.98 1.05 1.11; 1.03 1.06 1.13 1.18; 0.99 1.02 1.05 1.10; - - 1.00 1.07 / 0.93 0.93 1.02 1.03; 0.95 0.99 1.03 1.05
//   wide, one and 148 queries at ef 101, 110, 128, 200:  60 000 x 300 0.92 0.94 0.95 1.07, 0.94 0.94 0.99 1.23;  30 000 x 800 f16 0.98 1.02 1.08 1.24, 0.98 1.00 1.02 1.14
constexpr int kHandfulFrom = 72, kFewFrom = 56, kSomeFromLong = 80, kWideFrom = 140;
constexpr int kLongNarrow = 200, kLongWide = 250;  // smallest ef of a long walk
// The walks that count are those of the searches that take turns with this one on other streams as well (p.beside): a CTA of 16
// warps fills the registers of an SM, three of eight warps do, and what comes next waits.  32 batches through four streams, ms, by
// the batch alone / by all: 1.18 M x 50, 148 queries each, ef 64 and 200: 3.25 / 1.97 and 5.00 / 3.52; 444: 3.33 / 2.53 and 5.73 / 4.90; 300 000 x 96
// f16, 148: 2.95 / 1.54 and 4.50 / 2.66.  Four or more that take turns keep the chip full either way, so three CTAs of eight warps
// do up to six per SM (10 batches of 148 and 200 of 1.18 M x 50, ef 100: 1.12 and 1.11 times as fast as on the list, six and ten of 250 1.04 and 1.13, but
// 0.91 to 0.94 at ef 60 and on 128 floats); three batches of 200 at once do not fit (0.90).  fp32 rows above 64 values gain by 16
// warps up to 1.4 per SM in turn (32 batches of 50 of 300 000 x 128, 300 000 x 80 and 600 000 x 110, ef 200: 1.09, 1.19 and 1.15 times as fast as on the list
// with 8, 1.25, 1.25 and 1.34 with 16); three batches of 74 at once would not (0.83 to 0.91 at ef 100).  What 100 of them gain steadily with 16 (ef 350:
// 1.38 against 1.15 on 128 floats) they lose in a burst of three (ef 100: 0.80 against 1.08).
// kCtas: how many CTAs of four warps on a list an SM is to hold, said to the compiler, whose own count of registers moves with
// every change around it: seven of rows up to 64 values, six of up to 96.  ms, so / as it came out: 1000 queries of 200 000 x 32, ef 64
// and 100, 0.219 / 0.264 and 0.301 / 0.346 (six CTAs); 3000 of 300 000 x 64, ef 128 and 180, 0.588 / 0.625 and 0.714 / 0.764 (72 registers, six in
// shared memory); 2000 of 300 000 x 96, ef 100 and 128, 0.521 / 0.607 and 0.569 / 0.636 (five).
template <class Dist, int kCtas, int kFrontierCtas>
cudaError_t launch_walk_narrow(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  const long long walks = p.nq + p.beside;
  const bool long_rows = p.g.d > 64 && !p.g.rows16;
  const bool few = long_rows && p.beside > 0 ? 5 * walks <= 7ll * sm_count : walks <= sm_count;
  if (p.ef >= (walks <= 8 ? kHandfulFrom : kFewFrom) && few)
    return launch_frontier_t<Dist, 16, 16, 1>(p, 8192, sm_count, stream, sched);
  const bool some = walks <= (long long)sm_count * 3 || (p.beside >= 3 * p.nq && walks <= (long long)sm_count * 6);
  if (p.ef >= (long_rows ? kSomeFromLong : kFewFrom) && walks > sm_count && some)
    return launch_frontier_t<Dist, 8, 8, 3>(p, 8192, sm_count, stream, sched);
  if (p.ef <= kShortWalk) return launch_walk_t<Dist, 4, 4, kCtas>(p, 8192, sm_count, stream, sched);
  if (p.ef >= kLongNarrow && p.g.d > 32 && p.nq <= (long long)sm_count * 14 && walks <= (long long)sm_count * 20)
    return launch_frontier_t<Dist, 4, 8, kFrontierCtas>(p, 8192, sm_count, stream, sched);
  if (p.nq <= (long long)sm_count * 27) return launch_walk_t<Dist, 4, 8, kCtas>(p, 8192, sm_count, stream, sched);
  return launch_walk_t<Dist, 2, 8, 10>(p, 8192, sm_count, stream, sched);
}
// Wide rows, list / frontier: one of 150 000 x 960, ef 300 0.326 / 0.253 (16 x 16); 300 of them 0.890 / 0.679 (8 x 8); one and 148 of 200 000 x
// 200, ef 1500 1.44 / 0.93 and 3.28 / 1.48; with ef 25 and 10 the frontier is the slower one by 6 to 20 %, with ef 100 they are equal
// (300 000 x 300).  4 x 8: 1000 of 120 000 x 960, ef 200 0.75 / 0.76, ef 300 1.09 / 0.96, ef 400 1.45 / 1.22; of 300 000 x 300 0.73 / 0.74, 1.01 / 0.94,
// 1.28 / 1.12; of 200 000 x 150 f16 0.75 / 0.71, 0.94 / 0.81, 1.26 / 0.98; 600 of them, ef 1000 2.62 / 1.78; 400 of 120 000 x 960, ef 200 0.59 / 0.61.
template <class Dist>
cudaError_t launch_walk_wide(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  const bool brief = p.ef <= kShortWalk;
  const bool frontier = p.ef >= (p.g.d > 512 ? kShortWalk + 1 : kWideFrom);
  const long long walks = p.nq + p.beside;
  if (frontier && walks <= sm_count) return launch_frontier_t<Dist, 16, 16, 1>(p, 16384, sm_count, stream, sched);
  // while two CTAs of eight warps per SM hold all queries at once; further on four CTAs of four serve more (60 000 x 960, 2,
  // 3 and 4 queries per SM, four / eight warps: ef 100 1.21 1.06 0.94, ef 200 1.12 0.96 0.78, ef 400 1.12 0.92 0.73)
  if (p.nq <= (long long)sm_count * 2)
    return frontier ? launch_frontier_t<Dist, 8, 8, 2>(p, 16384, sm_count, stream, sched)
                    : launch_walk_t<Dist, 8, 8, 2>(p, 16384, sm_count, stream, sched);
  if (brief) return launch_walk_t<Dist, 4, 4, 4>(p, 16384, sm_count, stream, sched);
  if (p.ef >= kLongWide) return launch_frontier_t<Dist, 4, 8, 4>(p, 16384, sm_count, stream, sched);
  return launch_walk_t<Dist, 4, 8, 4>(p, 16384, sm_count, stream, sched);
}

template <class Row>
cudaError_t launch_search_walk(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  using E = Pick<Row>;
  const int d = p.g.d;
  if (d <= 32) return launch_walk_narrow<typename E::D32, 7, 6>(p, sm_count, stream, sched);
  if (d <= 64) return launch_walk_narrow<typename E::D64, 7, 6>(p, sm_count, stream, sched);
  if (d <= 96) return launch_walk_narrow<typename E::D96, 6, 5>(p, sm_count, stream, sched);
  if (d <= 128) return launch_walk_narrow<typename E::D128, 5, 5>(p, sm_count, stream, sched);
  // a warp gets one to five rows of a round: two rows of eight columns in flight bring a 3840-byte row in one round trip;
  // rows of up to four columns have nothing for the other four to load (300 000 x 300: 0.62 against 0.73 ms)
  if (d <= 512) return launch_walk_wide<typename E::Wide>(p, sm_count, stream, sched);
  return launch_walk_wide<typename E::Team>(p, sm_count, stream, sched);
}

}  // namespace hnsw
