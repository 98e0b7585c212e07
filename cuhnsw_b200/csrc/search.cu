// Batch kNN search over a device-resident graph: greedy descent through the upper layers and the
// ef_search-bounded layer-0 search in ONE launch (knn_search_kernel), or, for batches that need more
// than one wave of warps, a descent kernel, a sort of the queries by entry distance and the same search
// kernel serving the farthest entries first (entry_kernel, schedule_search).
//
// Replaces GetEntryPointsKernel + SearchGraphKernel and their host driver
// (cpp/include/cuda_search_kernels.cuh:11-165, cpp/src/cuhnsw_build.cu:210-290),
// which re-flatten and re-upload the graph on every call, launch once per
// layer and keep the heap in global memory.
#include <algorithm>

#include <cub/block/block_radix_sort.cuh>
#include <cub/device/device_radix_sort.cuh>

#include "kernels.h"
#include "beam.cuh"

namespace hnsw {

constexpr int kWarpsPerCta = 2;

// kEntries: the batch has been scheduled, every query's descent has ended at entry_node / entry_dist.  An instance of its
// own because the walk is cheaper without the descent beside it: 315 against 367 warp instructions per expansion by the
// counters (20 000 queries, 600 000 x 50, ef 200: 1.76 against 1.94 ms).
template <class Dist, class Table, bool kReverse, bool kEntries>
__global__ void __launch_bounds__(kWarpsPerCta * 32, Dist::kSearchMinCtas)
knn_search_kernel(SearchParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* mine = smem + (size_t)warp * p.smem_per_warp;
  Dist de;
  const VecTable tab = make_table(p.g);
  de.init(tab, mine);
  WarpList<Table> wl;
  wl.bind(mine + Dist::smem_bytes(p.g.d), p.ef, p.vsize, p.g.n);
  WalkCounters wc{0, 0, 0, 0};

  for (;;) {
    long long qi = 0;
    if (lane == 0) qi = (long long)atomicAdd(p.ticket, 1ull);
    qi = __shfl_sync(FULL, qi, 0);
    if (qi >= p.nq) break;
    if (p.order) qi = __shfl_sync(FULL, __ldg(p.order + qi), 0);
    de.load_query(p.queries + (size_t)qi * p.g.d);
    wl.reset();
    int cur;
    float dcur;
    if (kEntries) {
      cur = __shfl_sync(FULL, __ldg(p.entry_node + qi), 0);
      dcur = __shfl_sync(FULL, __ldg(p.entry_dist + qi), 0);
    } else {
      cur = p.g.enter_point;
      dcur = de.eval(cur, 1);
      dcur = __shfl_sync(FULL, dcur, 0);
      wc.evals += 1;
      greedy_descent(de, p.g.rowsU, p.g.strideU, p.g.upper_base, p.g.max_level, 0, cur, dcur, wc);
    }
    // layer 0: list = {entry}, visited = {entry} (cuda_search_kernels.cuh:108-112)
    wl.seed(mkkey(dcur, cur));
    wl.mark(cur);
    if (kReverse) beam_layer_reverse(de, wl, p.g.rows0, p.g.stride0, p.g.upper_base, 0, -1, wc);
    else beam_layer(de, wl, p.g.rows0, p.g.stride0, p.g.upper_base, 0, -1, wc);
    // ascending top-k, found = min(size, k); slots past `found` read -1 / +inf
    int found = min(wl.size, p.topk);
    for (int j = lane; j < p.topk; j += 32) {
      int id = -1;
      float dist = __int_as_float(0x7f800000);
      if (j < found) {
        unsigned long long k = wl.key(j);
        id = key_id(k);
        dist = key_dist(k);
        if (p.labels) id = __ldg(p.labels + id);
      }
      p.out_ids[(size_t)qi * p.topk + j] = id;
      p.out_dist[(size_t)qi * p.topk + j] = dist;
    }
    if (lane == 0) p.out_found[qi] = found;
    __syncwarp();
  }
  if (p.stats && lane == 0) {
    atomicAdd(p.stats + 0, (unsigned long long)wc.evals);
    atomicAdd(p.stats + 1, (unsigned long long)wc.expansions);
    atomicAdd(p.stats + 2, (unsigned long long)wc.sweeps);
    atomicAdd(p.stats + 3, (unsigned long long)wc.inserts);
  }
}

// First stage of a scheduled search: one warp per query walks down the upper layers
// (GetEntryPointsKernel of the reference, cuda_search_kernels.cuh:11-77, all layers in one launch) and
// leaves where it ended, how far that is, and a sort key that puts the farthest entries first.
template <class Dist>
__global__ void __launch_bounds__(kWarpsPerCta * 32) entry_kernel(SearchParams p, SearchSchedule s) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long qi = (long long)blockIdx.x * kWarpsPerCta + warp;
  if (qi >= p.nq) return;
  Dist de;
  const VecTable tab = make_table(p.g);
  de.init(tab, smem + (size_t)warp * Dist::smem_bytes(p.g.d));
  WalkCounters wc{0, 0, 0, 0};
  de.load_query(p.queries + (size_t)qi * p.g.d);
  int cur = p.g.enter_point;
  float dcur = de.eval(cur, 1);
  dcur = __shfl_sync(FULL, dcur, 0);
  wc.evals += 1;
  greedy_descent(de, p.g.rowsU, p.g.strideU, p.g.upper_base, p.g.max_level, 0, cur, dcur, wc);
  if (lane == 0) {
    s.entry_node[qi] = cur;
    s.entry_dist[qi] = dcur;
    // sort key: farthest entry first.  Small batches are sorted by one CTA (sort_schedule_kernel), which wants
    // the query number in the low half of the word.
    const unsigned key = ~f2ord(dcur);
    if (p.nq <= kBlockSortMax) {
      s.keys[qi] = (key & 0xffff0000u) | (unsigned)qi;
    } else {
      s.keys[qi] = key;
      s.index[qi] = (int)qi;
    }
    if (p.stats) {
      atomicAdd(p.stats + 0, (unsigned long long)wc.evals);
      atomicAdd(p.stats + 2, (unsigned long long)wc.sweeps);
    }
  }
}

template <class Dist>
static cudaError_t launch_entry_t(const SearchParams& p, const SearchSchedule& s, cudaStream_t stream) {
  const size_t smem = Dist::smem_bytes(p.g.d) * kWarpsPerCta;
  auto kern = entry_kernel<Dist>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const long long grid = (p.nq + kWarpsPerCta - 1) / kWarpsPerCta;
  kern<<<(unsigned)grid, kWarpsPerCta * 32, smem, stream>>>(p, s);
  return cudaGetLastError();
}

template <class Row>
static cudaError_t launch_entry_rows(const SearchParams& p, const SearchSchedule& s, cudaStream_t stream) {
  using E = Pick<Row>;
  const int d = p.g.d;
  return d <= 32    ? launch_entry_t<typename E::D32>(p, s, stream)
         : d <= 64  ? launch_entry_t<typename E::D64>(p, s, stream)
         : d <= 96  ? launch_entry_t<typename E::D96>(p, s, stream)
         : d <= 128 ? launch_entry_t<typename E::D128>(p, s, stream)
                    : launch_entry_t<typename E::Wide>(p, s, stream);
}

// Orders up to kBlockSortMax packed words (sort key in the upper 16 bits, query number in the lower 16) with one
// CTA: a block-wide radix sort over the key bits, stable, so equal keys stay in query order.  Writes the query
// numbers in sorted order.
constexpr int kBlockSortThreads = 1024, kBlockSortItems = 10;
__global__ void __launch_bounds__(kBlockSortThreads) sort_schedule_kernel(const unsigned* __restrict__ words, int nq,
                                                                          int* __restrict__ order) {
  using Sort = cub::BlockRadixSort<unsigned, kBlockSortThreads, kBlockSortItems>;
  __shared__ typename Sort::TempStorage tmp;
  unsigned mine[kBlockSortItems];
#pragma unroll
  for (int i = 0; i < kBlockSortItems; ++i) {
    const int at = threadIdx.x * kBlockSortItems + i;
    mine[i] = at < nq ? words[at] : 0xffffffffu;
  }
  Sort(tmp).Sort(mine, 16, 32);
#pragma unroll
  for (int i = 0; i < kBlockSortItems; ++i) {
    const int at = threadIdx.x * kBlockSortItems + i;
    if (at < nq) order[at] = (int)(mine[i] & 0xffffu);
  }
}

size_t search_schedule_tmp_bytes(long long nq) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                  (int*)nullptr, (int)nq, 16, 32);
  return bytes;
}

cudaError_t schedule_search(SearchParams& p, const SearchSchedule& s, cudaStream_t stream) {
  if (p.nq > s.capacity || p.nq > 0x7fffffffll) return cudaErrorInvalidValue;  // the sort counts items in an int
#define CALL(R) launch_entry_rows<R>(p, s, stream)
  cudaError_t e = HNSW_WITH_ROWS(p.g.rows16, CALL);
#undef CALL
  if (e != cudaSuccess) return e;
  // the upper 16 bits of the key (sign, exponent, 7 bits of mantissa) order the queries finely enough
  if (p.nq <= kBlockSortMax) {
    sort_schedule_kernel<<<1, kBlockSortThreads, 0, stream>>>(s.keys, (int)p.nq, s.order);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    p.order = s.order;
    p.entry_node = s.entry_node;
    p.entry_dist = s.entry_dist;
    return cudaSuccess;
  }
  size_t bytes = s.sort_tmp_bytes;
  e = cub::DeviceRadixSort::SortPairs(s.sort_tmp, bytes, (const unsigned*)s.keys, s.keys_sorted, (const int*)s.index,
                                      s.order, (int)p.nq, 16, 32, stream);
  if (e != cudaSuccess) return e;
  p.order = s.order;
  p.entry_node = s.entry_node;
  p.entry_dist = s.entry_dist;
  return cudaSuccess;
}

template <class Dist, class Table, bool kReverse>
static cudaError_t launch_search_tr(const SearchParams& p0, int sm_count, cudaStream_t stream,
                                    const SearchSchedule* sched);

template <class Dist, class Table>
static cudaError_t launch_search_tt(const SearchParams& p0, int sm_count, cudaStream_t stream,
                                    const SearchSchedule* sched) {
  return p0.reverse_cand ? launch_search_tr<Dist, Table, true>(p0, sm_count, stream, sched)
                         : launch_search_tr<Dist, Table, false>(p0, sm_count, stream, sched);
}

// Which visited table: by row type (Dist::kTwoTags, kTwoTagsInside), but two tags per bucket also where four would need 32 bits each and two do
// not: one factor of two of the number of rows, 16.8 to 33.5 M with 2048 entries, whose 4 KB would hold 1024.  17 M x 16, 10 000
// queries, ef 200 and 300, and 40 000, ef 200: 1.35, 1.94 and 3.81 ms with 1024 entries of 32 bits, 1.31, 1.86 and 3.68 so.
template <class Dist>
static cudaError_t launch_search_t(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  if constexpr (!Dist::kTwoTags) {
    if (!VisitedTable::needs_wide(p.vsize, p.g.n) || VisitedPairs::needs_wide(p.vsize, p.g.n))
      return launch_search_tt<Dist, VisitedTable>(p, sm_count, stream, sched);
  }
  return launch_search_tt<Dist, VisitedPairs>(p, sm_count, stream, sched);
}

// CTAs of a search kernel that an SM holds
template <class K>
static cudaError_t residents(K kern, size_t smem, int* per_sm) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, kWarpsPerCta * 32, smem);
  return e != cudaSuccess ? e : *per_sm < 1 ? cudaErrorInvalidConfiguration : cudaSuccess;
}

template <class Dist, class Table, bool kReverse>
static cudaError_t launch_search_tr(const SearchParams& p0, int sm_count, cudaStream_t stream,
                                    const SearchSchedule* sched) {
  SearchParams p = p0;
  const auto smem_of = [&](size_t list) { return (Dist::smem_bytes(p.g.d) + list + 15) / 16 * 16; };
  using Inside = std::conditional_t<Dist::kTwoTagsInside, VisitedPairs, Table>;
  p.smem_per_warp = (int)smem_of(WarpList<Inside>::smem_bytes(p.ef, p.vsize, p.g.n));
  size_t smem = (size_t)p.smem_per_warp * kWarpsPerCta;
  int per_sm = 0;
  cudaError_t e = residents(knn_search_kernel<Dist, Inside, kReverse, false>, smem, &per_sm);
  if (e != cudaSuccess) return e;
  const long long want = (p.nq + kWarpsPerCta - 1) / kWarpsPerCta;
  long long grid = std::max(1ll, std::min((long long)per_sm * sm_count, want));
  e = cudaMemsetAsync(p.ticket, 0, sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return e;
  // more queries than resident warps: start the long walks first
  if (sched && p.nq > grid * kWarpsPerCta && p.nq <= sched->capacity && p.nq <= 0x7fffffffll) {
    e = schedule_search(p, *sched, stream);
    if (e != cudaSuccess) return e;
    p.smem_per_warp = (int)smem_of(WarpList<Table>::smem_bytes(p.ef, p.vsize, p.g.n));
    smem = (size_t)p.smem_per_warp * kWarpsPerCta;
    e = residents(knn_search_kernel<Dist, Table, kReverse, true>, smem, &per_sm);
    if (e != cudaSuccess) return e;
    grid = std::max(1ll, std::min((long long)per_sm * sm_count, want));
    knn_search_kernel<Dist, Table, kReverse, true><<<(unsigned)grid, kWarpsPerCta * 32, smem, stream>>>(p);
  } else {
    knn_search_kernel<Dist, Inside, kReverse, false><<<(unsigned)grid, kWarpsPerCta * 32, smem, stream>>>(p);
  }
  return cudaGetLastError();
}

// (the same for both tables where one of them is chosen: 16 bits per entry if two tags per bucket can do with that, else 32)
size_t search_smem_per_cta(int d, int ef, int vsize, long long n) {
  size_t dq = d <= 128 ? 0 : DistLarge::smem_bytes(d);
  size_t per_warp = (dq + WarpList<VisitedPairs>::smem_bytes(ef, vsize, n) + 15) / 16 * 16;
  return per_warp * kWarpsPerCta;
}

// One CTA per query while that is the faster way: up to so many queries per SM, which no rule on sizes hits for all data.
// Measured with tables of 200 000 to 300 000 rows, time of one CTA / one warp per query (device buffers, medians of nine
// launches, L2 cache emptied before each):
//   short walks end before rounds and, from a wave on, the entry kernel and the sort pay: 300 000 x 50, 6 and 8 queries per
//   SM: ef 10 0.86 and 0.88, ef 30 0.83 and 0.81, ef 50 0.81 and 0.80 (the line is at 6 below ef 40, at 14 above: ef 100, 12 and
//   24 per SM, 0.82 and 0.98); fp32 rows of 65 values and more, whose evaluations four warps share, hold out longer: 300 000 x 128,
//   12 and 20: ef 20 0.82 and 1.10, ef 50 0.70 and 0.92; 16 links x 96, 20 per SM, 0.96 at ef 40.
//   walks of 200 to 400: 300 000 x 50, 28 and 36 per SM, 0.91 and 1.06 at ef 200 (44: 1.23), 0.81 and 1.03 at 400; x 128, ef 200, 0.79 and
//   0.96; 16 links x 96, ef 300, 0.74 and 0.95; rows of up to 32 values: 32 links, ef 250, 8, 12 and 18 per SM 0.68 0.73 0.77, 20 links at 20
//   0.80, 16 links, ef 300, 28 and 36 0.88 and 1.02.
//   long lists leave an SM 4 to 8 CTAs: 300 000 x 128, 14 and 26 per SM: ef 600 0.54 and 1.07, ef 800 0.52 and 1.15, ef 1200 0.63 and 1.48;
//   24 links x 50, ef 1200, 12 and 20: 0.57 and 1.06; ef 1000, 14 and 24 per SM: 20 links x 48 0.57 and 0.93, 32 links x 48 0.62 and 1.07.
//   Once a list is so long that hardly more warps than CTAs fit either: ef 4800, 20 and 36 per SM, 1.02 and 1.08.
static int narrow_walks_per_sm(int d, int rows16, int links, int ef) {
  const bool long_rows = d > 64 && !rows16, many_links = links > 24;
  if (ef >= 4000) return 36;
  if (ef < 40) return long_rows ? (ef < 16 ? 4 : 14) : 6;
  if (d <= 32 && links > 16) return std::min({16, std::max(8, ef / 8), 11000 / ef});
  const int few = d <= 32 ? ef / 5 : std::max(14, ef * 27 / 128);
  const int many = d <= 64 ? (many_links ? 11000 : 15000) / ef
                           : long_rows && ef >= 2000 ? 24 : std::max(14, 14000 / ef);
  return std::min({d <= 64 && many_links ? 30 : 36, few, many});
}
// Wide rows: warps keep 16 float4 in flight each and win once 8 to 16 of them fill an SM; when, depends on the data more than
// on the sizes.  One CTA / one warp per query at 7, 8 and 10 queries per SM: 100 000 x 200: ef 250 0.93 1.03 1.16, ef 400 0.90
// 1.04 1.17, ef 700 0.97 1.09 1.24, ef 3000 0.56 0.59 0.73; 200 000 x 150: ef 250 0.74 0.78 0.80, ef 400 0.73 0.80 0.80, ef 700
// 0.67 0.77 0.86.  60 000 x 960 at 10 and 14: ef 50 0.85 0.84, ef 200 1.03 1.16, ef 400 0.85 1.03, ef 1600 0.64 0.75.
static int wide_walks_per_sm(int d, int ef) {
  if (d > 512) return ef > 200 && ef < 1200 ? 10 : 14;
  return ef > 300 && ef < 2000 ? 7 : 10;
}
// Otherwise one warp per query; for few queries over rows above 512 floats with 32 float4 loads in flight instead of 16
// (60 000 x 960, 8 and 10 queries per SM: ef 100 0.84 and 0.89, ef 400 0.77 and 1.12).  Expanding the farthest key first
// knows no next nodes to prepare: always one warp.
int search_kernel_kind(int d, int rows16, int links, int ef, long long nq, int team, int reverse_cand, int sm_count) {
  const int walks = d <= 128 ? narrow_walks_per_sm(d, rows16, links, ef) : wide_walks_per_sm(d, ef);
  if (!reverse_cand && (team == 1 || (team < 0 && nq <= (long long)sm_count * walks))) return kSearchTeam;
  if (d <= 128) return kSearchWarpSmall;
  return d > 512 && nq <= (long long)sm_count * 10 ? kSearchWarpDeep : kSearchWarp;
}

template <class Row>
static cudaError_t launch_search_rows(const SearchParams& p, int sm_count, cudaStream_t stream,
                                      const SearchSchedule* sched) {
  using E = Pick<Row>;
  const int d = p.g.d;
  if (d <= 32) return launch_search_t<typename E::D32>(p, sm_count, stream, sched);
  if (d <= 64) return launch_search_t<typename E::D64>(p, sm_count, stream, sched);
  if (d <= 96) return launch_search_t<typename E::D96>(p, sm_count, stream, sched);
  if (d <= 128) return launch_search_t<typename E::D128>(p, sm_count, stream, sched);
  if (search_kernel_kind(d, p.g.rows16, p.g.stride0, p.ef, p.nq, p.team, p.reverse_cand, sm_count) == kSearchWarpDeep)
    return launch_search_t<typename E::WideDeep>(p, sm_count, stream, sched);
  return launch_search_t<typename E::Wide>(p, sm_count, stream, sched);
}

cudaError_t launch_search(const SearchParams& p, int sm_count, cudaStream_t stream, const SearchSchedule* sched) {
  if (p.nq <= 0) return cudaSuccess;
  if (search_kernel_kind(p.g.d, p.g.rows16, p.g.stride0, p.ef, p.nq, p.team, p.reverse_cand, sm_count) == kSearchTeam)
    return p.g.rows16 == kRowsF16    ? launch_search_walk_f16(p, sm_count, stream, sched)
           : p.g.rows16 == kRowsBF16 ? launch_search_walk_bf16(p, sm_count, stream, sched)
                                     : launch_search_walk_f32(p, sm_count, stream, sched);
#define CALL(R) launch_search_rows<R>(p, sm_count, stream, sched)
  return HNSW_WITH_ROWS(p.g.rows16, CALL);
#undef CALL
}

}  // namespace hnsw

// ---------------------------------------------------------------------------
// Search that allocates nothing
// ---------------------------------------------------------------------------
// Some callers must not reach cudaMalloc: a serving process that has already handed every free byte of
// device memory to its own pool allocator (a late cudaMalloc there fails or evicts), a job running under a
// fixed memory budget, or a real-time loop that cannot take the device-wide synchronisation cudaMalloc and
// cudaFree imply.  For them the staging buffers and the work ticket of the search kernel live in one
// file-scope device array of fixed size instead of grow-on-demand allocations.  Every GPU that loads this
// library carries the array (4 MiB) until the process exits.
//
// In host code the name `g_search_scratch` is only the runtime's handle of the symbol, not a device address:
// a kernel given `g_search_scratch` from the host would fault or, where the GPU can reach host memory, use the
// wrong memory.  The device address is obtained once per device with cudaGetSymbolAddress (with that device
// current) and it is that pointer that is handed to the kernel.
#include <mutex>

namespace hnsw {

constexpr size_t kStaticScratchBytes = 4u << 20;
constexpr int kMaxDevices = 64;
static __device__ __align__(256) unsigned char g_search_scratch[kStaticScratchBytes];

static std::mutex g_scratch_mu;
static void* g_scratch_addr[kMaxDevices] = {};

static cudaError_t static_scratch_address(unsigned char** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_addr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_search_scratch);  // set-up: first call on this device
    if (e != cudaSuccess) return e;
    g_scratch_addr[dev] = p;
  }
  *out = static_cast<unsigned char*>(g_scratch_addr[dev]);
  return cudaSuccess;
}

static size_t align256(size_t x) { return (x + 255) / 256 * 256; }

size_t search_static_capacity() { return kStaticScratchBytes; }

size_t search_static_bytes(long long nq, int d, int topk) {
  return 256 + align256((size_t)nq * d * sizeof(float)) + 2 * align256((size_t)nq * topk * 4) +
         align256((size_t)nq * sizeof(int));
}

// Host buffers in and out; the caller has checked search_static_bytes() <= search_static_capacity().
// Layout of the array: [ticket | queries | ids | distances | found].  Only the ticket has to start at zero and
// the launcher clears it on the stream; everything else is overwritten before it is read.  The array is shared
// by every call in the process on this device, so two calls that overlap on the GPU race on it.
cudaError_t search_static(const SearchParams& proto, const float* h_queries, int* h_ids, float* h_dist, int* h_found,
                          int sm_count, cudaStream_t stream) {
  unsigned char* base = nullptr;
  cudaError_t e = static_scratch_address(&base);
  if (e != cudaSuccess) return e;
  const long long nq = proto.nq;
  const size_t qbytes = (size_t)nq * proto.g.d * sizeof(float), rbytes = (size_t)nq * proto.topk * 4;
  SearchParams p = proto;
  p.ticket = reinterpret_cast<unsigned long long*>(base);
  p.stats = nullptr;
  unsigned char* at = base + 256;
  float* d_q = reinterpret_cast<float*>(at);
  at += align256(qbytes);
  p.out_ids = reinterpret_cast<int*>(at);
  at += align256(rbytes);
  p.out_dist = reinterpret_cast<float*>(at);
  at += align256(rbytes);
  p.out_found = reinterpret_cast<int*>(at);
  p.queries = d_q;
  if ((e = cudaMemcpyAsync(d_q, h_queries, qbytes, cudaMemcpyHostToDevice, stream)) != cudaSuccess) return e;
  if ((e = launch_search(p, sm_count, stream)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(h_ids, p.out_ids, rbytes, cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(h_dist, p.out_dist, rbytes, cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(h_found, p.out_found, (size_t)nq * sizeof(int), cudaMemcpyDeviceToHost, stream)) !=
      cudaSuccess)
    return e;
  return cudaStreamSynchronize(stream);
}

}  // namespace hnsw
