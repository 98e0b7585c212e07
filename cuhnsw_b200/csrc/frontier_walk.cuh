// The graph walk of one CTA per query for few queries and for long walks, on a Frontier instead of a list of the ef closest
// keys.
//
// Rounds as in walk.cuh: select up to P unexpanded nodes, prepare them together, commit those whose turn it is.  There every
// commit ends in a merge into the sorted list, 1500 cycles of one warp, half to two thirds of a round.  Here
//   select   reads the first keys of the front: a register per lane,
//   commit   decides for all prepared nodes at once how many are expanded one behind the other (what each of them brings
//            at best is known from its evaluation), and takes what they bring in 32 neighbours at a time, whichever node
//            they belong to.
// Nothing a prepared node brings is seen by the frontier or the visited table before its commit, so keys, visited
// nodes and results are those of the literal walk, step for step.
//
// Bound: the chain of a round, two memory round trips and a commit of about 2500 cycles.  One B200, ms of device time with the L2 cache
// emptied before each launch, with the list / so: one query of 100 000 x 50, ef 300: 0.261 / 0.181; 148 of 1.18 M x 50, ef 200: 0.477 / 0.350; 37 of 1 M x 96 bfloat16, ef 128: 0.302 / 0.256;
// one of 150 000 x 960, ef 300: 0.326 / 0.253.  It helps the more the longer the list would be (1500 keys: 1.5 to 2.3 times as fast), and the
// less the more neighbours a node brings, as a commit costs by the neighbour and a merge by the key that is close enough
// (search_walk.cuh).
#pragma once
#include "frontier.cuh"
#include "walk.cuh"

namespace hnsw {

// What the warps of one walk tell each other, in shared memory: 32-bit words at these offsets.
template <int P>
struct FrontierBoard {
  static constexpr int kOp = 0, kNodes = 4, kPool = 8, kQuery = 12;  // operation, nodes of the round, rows in the pool, query
  static constexpr int kNode = 16;              // P pairs: node id, address and (upper 8 bits) number of its buffer
  static constexpr int kCount = kNode + 8 * P;  // new neighbours of each
  static constexpr int kLeast = kCount + 4 * P; // of each of the 2 P buffers, the smallest distance image
  static constexpr int kBytes = (kLeast + 8 * P + 15) / 16 * 16;
};

template <class Dist, int W, int P>
struct FrontierWalk {
  static constexpr int kBuffers = 2 * P;
  static_assert(W > 1 && kBuffers <= 32, "a lane stands for a buffer");
  // Front keys that are prepared.  More than P of them evaluate more for nothing (8 nodes, 1.33 evaluations for each distinct
  // row among the first 16, 1.26 among the first 8, in 6 % more rounds).
  static constexpr int kWindow = P > 8 ? 16 : P;
  static constexpr int kMost = kBuffers < 31 ? kBuffers : 31;  // nodes that are committed at once
  // a front key's tag: -1, or the buffer that holds the node's new neighbours and, from this bit on, their number
  static constexpr int kCountAt = 8;
  using Board = FrontierBoard<P>;

  Dist de;
  Frontier fr;  // keys: warp 0; the visited table: all
  unsigned found;  // shared-memory address of kBuffers x stride keys: the prepared nodes' new neighbours
  unsigned pool;   // of the rows to evaluate: (id, place of the key in `found`: address and, in a round, buffer)
  unsigned board;
  LayerRows rows;    // of the searched layer
  int stride, self;  // slots of an adjacency row (= keys per buffer); node to leave out, or -1
  int lane;
  unsigned lower;  // lanes below this one
  WalkCounters wc;

  // shared memory of one walk, without the distance engine's own
  __host__ __device__ static size_t smem_bytes(int slots, int stride, int entries, long long n) {
    return (Frontier::smem_bytes(slots) + VisitedTable::smem_bytes(entries, n) + (size_t)kBuffers * stride * 8 +
            (size_t)P * stride * 8 + Board::kBytes + 15) / 16 * 16;
  }
  __device__ __forceinline__ void bind(unsigned char* smem, int ef, int slots, int stride_, int entries, long long n) {
    unsigned at = kept(smem_addr(smem));
    fr.bind(at, ef, slots, entries, n);
    found = at += Frontier::smem_bytes(slots) + fr.vbytes;
    pool = at += kBuffers * stride_ * 8;
    board = at + P * stride_ * 8;
    stride = stride_;
    lane = lane_number();
    lower = (1u << lane) - 1u;
    wc = WalkCounters{0, 0, 0, 0};
  }
  static __device__ __forceinline__ int warp() { return __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0); }
  __device__ __forceinline__ unsigned place_of(int buffer) const { return found + 8 * stride * buffer; }
  // a word of the board, known to be the same in every lane
  __device__ __forceinline__ int posted(int at) const { return __shfl_sync(FULL, (int)lds32(board + at), 0); }

  // ---- parts every warp of the walk takes ----

  // Adjacency rows of `count` nodes, whose neighbours go to the buffers at `place`: those the visited table does not know
  // go to the pool, the number of those of node i to have[i].  The table is only read here; nodes enter it when
  // their key is committed.
  template <int N>
  __device__ __forceinline__ void filter_rows(const int (&node)[N], const unsigned (&place)[N], int count,
                                              int (&have)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) have[i] = 0;
    for (int base = 0; base < stride; base += 32) {
      int nid[N];
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i < count) nid[i] = rows.read(rows.row(node[i]), base);
      unsigned m[N];
      int all = 0, at = 0;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        m[i] = 0u;
        if (i < count) {
          const bool known = fr.knows(nid[i]);
          m[i] = __ballot_sync(FULL, nid[i] >= 0 && nid[i] != self && !known);
          all += __popc(m[i]);
        }
      }
      if (lane == 0) at = (int)atomic_add_shared(board + Board::kPool, all);
      at = __shfl_sync(FULL, at, 0);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int before = __popc(m[i] & lower);
        if ((m[i] >> lane) & 1u) sts64(pool + 8 * (at + before), (unsigned)nid[i], place[i] + 8 * (have[i] + before));
        at += __popc(m[i]);
        have[i] += __popc(m[i]);
      }
    }
  }
  // this warp's share of the round on the board
  // (`words`: two of the board's in each lane)
  __device__ __forceinline__ uint2 board_words() const { return lds64(board + 8 * min(lane, 1 + P)); }
  __device__ __forceinline__ void filter_posted(int w, uint2 words) {
    constexpr int N = (P + W - 1) / W;
    const int nsel = __shfl_sync(FULL, (int)words.y, 0);
    if (w >= nsel) return;
    const int count = (nsel - w + W - 1) / W;
    int node[N], have[N];
    unsigned place[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int c = min(w + W * i, P - 1);
      node[i] = __shfl_sync(FULL, (int)words.x, 2 + c);
      place[i] = __shfl_sync(FULL, words.y, 2 + c);
    }
    filter_rows(node, place, count, have);
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < count && lane == 0) sts32(board + Board::kCount + 4 * (w + W * i), (unsigned)have[i]);
  }

  // Warps 1 .. W - 1: every operation starts and ends at a block barrier, as warp 0's do.  Returns, behind its first
  // barrier, the first operation that is not the walk's own.
  __device__ __forceinline__ int help(const float* queries) {
    const int w = warp();
    for (;;) {
      __syncthreads();
      const uint2 words = board_words();
      const int op = __shfl_sync(FULL, (int)words.x, 0);
      if (op == kWalkOver || op == kWalkKeys) return op;
      if (op == kWalkQuery || op == kWalkNode) {
        if (!Dist::kSharedQuery) load(op, queries);
        if (op == kWalkNode) self = posted(Board::kQuery);
        fr.clear(w, W);
      } else {
        if (op == kWalkRound) {
          filter_posted(w, words);
          __syncthreads();
        }
        de.template eval_pool<true>(pool, posted(Board::kPool), w, W, board + Board::kLeast);
      }
      __syncthreads();
    }
  }
  // the query whose number is on the board, or the stored row
  __device__ __forceinline__ void load(int op, const float* queries) {
    const long long qi = (unsigned)posted(Board::kQuery);
    if (op == kWalkQuery) de.load_query(queries + (size_t)qi * de.t.d);
    else de.load_query_row((int)qi);
  }

  // ---- warp 0 ----
  __device__ __forceinline__ void post(int op) {
    if (lane == 0) sts32(board + Board::kOp, op);
    __syncthreads();
  }
  // distances of the n rows in the pool
  __device__ __forceinline__ void evaluate_rows(int n) {
    if (lane == 0) sts32(board + Board::kPool, n);
    post(kWalkRows);
    de.template eval_pool<true>(pool, n, 0, W, board + Board::kLeast);
    __syncthreads();
    wc.evals += n;
  }
  // query `i` of `queries` (op kWalkQuery), or stored row i, which the walk then leaves out (kWalkNode)
  __device__ __forceinline__ void start(int op, const float* queries, long long i) {
    if (lane == 0) sts32(board + Board::kQuery, (unsigned)i);
    post(op);
    load(op, queries);
    if (op == kWalkNode) self = (int)i;
    fr.clear(0, W);
    __syncthreads();
  }
  __device__ __forceinline__ void finish() { post(kWalkOver); }

  // Greedy walk through layers top .. 1 (same rule as greedy_descent in beam.cuh).
  __device__ __forceinline__ void descend(const GraphView& g, int& cur, float& dcur) {
    cur = g.enter_point;
    if (lane == 0) sts64(pool, (unsigned)cur, found);
    evaluate_rows(1);
    dcur = ord2f(__shfl_sync(FULL, lds32(found), 0));  // (the shuffle tells the compiler that all lanes agree)
    if (g.max_level == 0) return;
    int first = __ldg(g.upper_base + cur);  // the node's row on layer 1
    for (int l = g.max_level; l > 0; --l) {
      for (;;) {
        const int* row = g.rowsU + ((size_t)first + (l - 1)) * g.strideU;
        wc.sweeps += 1;
        int n = 0, firsts[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < 2; ++c) {  // (at most 64 links)
          const int li = 32 * c + lane;
          const int nid = li < g.strideU ? __ldg(row + li) : -1;
          const unsigned m = __ballot_sync(FULL, nid >= 0);
          const int at = n + __popc(m & lower);
          if (nid >= 0) {
            sts64(pool + 8 * at, (unsigned)nid, found + 8 * at);
            firsts[c] = __ldg(g.upper_base + nid);  // (links are packed: entry 32 c + lane of the pool)
          }
          n += __popc(m);
        }
        if (n == 0) break;
        evaluate_rows(n);
        int best_id = cur, best_first = first;
        float best_d = dcur;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (32 * c >= n) break;
          uint2 k = 32 * c + lane < n ? lds64(found + 8 * (32 * c + lane)) : make_uint2(~0u, ~0u);
          if (k.x < f2ord(-__int_as_float(0x7f800000))) k.x = ~0u;  // a negative NaN is not closest
          const unsigned least = __reduce_min_sync(FULL, k.x);
          const int at = __ffs(__ballot_sync(FULL, k.x == least)) - 1;  // first in row order
          const int id = __shfl_sync(FULL, (int)k.y, at), next = __shfl_sync(FULL, firsts[c], at);
          if (ord2f(least) < best_d) {
            best_d = ord2f(least);
            best_id = id;
            best_first = next;
          }
        }
        __syncwarp();
        if (best_id == cur) break;
        cur = best_id;
        dcur = best_d;
        first = best_first;
      }
    }
  }

  // the walk's only key, and visited
  __device__ __forceinline__ void seed(int id, float dist) {
    fr.reset();
    fr.push_front(mkkey(dist, id));
    if (lane == 0) fr.test_and_set(id);
    __syncwarp();
  }

  // the keys are the neighbours in an adjacency row of the searched layer
  __device__ __forceinline__ void seed_row(int owner) {
    const int* row = rows.row(owner);
    fr.reset();
    int n = 0;
    for (int base = 0; base < stride; base += 32) {
      const int nid = rows.read(row, base);
      const bool on = nid >= 0 && nid != self;
      const unsigned m = __ballot_sync(FULL, on);
      const int at = n + __popc(m & lower);
      if (on) sts64(pool + 8 * at, (unsigned)nid, found + 8 * at);
      n += __popc(m);
    }
    if (n == 0) return;
    evaluate_rows(n);
    for (int base = 0; base < n; base += 32) {
      if (base > 0 && fr.short_of_room()) fr.compact();
      take_in(lds64(found + 8 * min(base + lane, n - 1)), base + lane < n, false);
    }
  }

  // Of the lanes that are `on`, the lowest one with each id.  Ten bits of a hash by ballots, then a look at the lane they
  // point to; only if that has another id, all ids are compared (__match_any_sync takes a step per different id).
  __device__ __forceinline__ bool first_of_its_kind(int id, bool on) const {
    const unsigned h = (unsigned)id * 2654435761u;
    unsigned m = __ballot_sync(FULL, on);
#pragma unroll
    for (int b = 22; b < 32; ++b) {
      const bool bit = (h >> b) & 1u;
      const unsigned with = __ballot_sync(FULL, bit);
      m &= bit ? with : ~with;
    }
    m &= lower;
    const int other = __shfl_sync(FULL, id, m ? __ffs(m) - 1 : lane);
    const bool like = on && m != 0u;
    bool earlier = like;
    if (__any_sync(FULL, like && other != id)) earlier = (__match_any_sync(FULL, on ? id : -1) & lower) != 0u;
    return on && !earlier;
  }
  // Up to 32 new neighbours (image, id), one per lane, of nodes that are being expanded: those that come for the first time
  // enter the visited table, and the frontier if they are close enough.  `several`: an id may come twice.
  __device__ __forceinline__ void take_in(uint2 v, bool have, bool several) {
    const VisitedTable::Seen seen = fr.enter((int)v.y, have);
    bool fresh = have && !seen.known;
    __syncwarp();
    fr.settle(seen, fresh);
    if (several) fresh = first_of_its_kind((int)v.y, fresh);
    const unsigned long long k = ((unsigned long long)v.x << 32) | v.y;
    fr.take(k, fresh, seen.full, wc);
    prefetch_row((int)v.y, fresh && k < fr.split && k < fr.limit);  // likely to be prepared in the next round
  }
  // an adjacency row of the searched layer on its way to the L2 cache (37 and 148 queries of 300 000 x 128, ef 200: 0.436 -> 0.421 and 0.481 ->
  // 0.464 ms, warm caches or not; a table that lies in the cache as a whole, 100 000 x 50, loses 1 to 2 %)
  __device__ __forceinline__ void prefetch_row(int id, bool on) const {
    const int* row = rows.row(on ? id : 0) - lane;
    prefetch_l2_if(on, row);
    prefetch_l2_if(on, row + stride - 1);
  }

  // Up to P nodes of the front that are not prepared yet are.
  __device__ __forceinline__ void prepare() {
    const bool open = fr.tag < 0 && lane < min(fr.near, kWindow);
    const unsigned om = __ballot_sync(FULL, open);
    const unsigned used = __reduce_or_sync(FULL, fr.tag >= 0 ? 1u << (fr.tag & (kBuffers - 1)) : 0u);
    // at least one buffer is free: every round commits the first key of the front, prepared in that round at the latest
    if (lane < kBuffers && !((used >> lane) & 1u)) sts32(fr.scratch + 4 * __popc(~used & lower), lane);
    const int nsel = min(min(P, kBuffers - __popc(used)), __popc(om));
    __syncwarp();
    const int rank = __popc(om & lower);
    const bool chosen = open && rank < nsel;
    const int buffer = (int)lds32(fr.scratch + 4 * (rank & (kBuffers - 1)));
    if (chosen) {
      sts64(board + Board::kNode + 8 * rank, (unsigned)fr.front, place_of(buffer) | (unsigned)buffer << 24);
      sts32(board + Board::kLeast + 4 * buffer, ~0u);
    }
    if (lane == 0) {
      sts32(board + Board::kNodes, nsel);
      sts32(board + Board::kPool, 0);
    }
    post(kWalkRound);
    filter_posted(0, board_words());
    __syncthreads();
    const int total = posted(Board::kPool);
    de.template eval_pool<true>(pool, total, 0, W, board + Board::kLeast);
    __syncthreads();
    if (chosen) fr.tag = buffer | ((int)lds32(board + Board::kCount + 4 * rank) << kCountAt);
    wc.evals += total;
  }

  // Commits the prepared nodes at the beginning of the front, until the first key is not a prepared one (true) or the walk
  // is over (false).  As many at once as possible: a node is expanded right behind those before it if it is closer than
  // everything that they bring (equal distances wait for their turn at the front, where the whole keys are compared), if
  // fewer than ef keys are expanded then, and if there is room for what it brings.  What they bring is then taken in 32
  // neighbours at a time, whichever node they belong to.
  __device__ __forceinline__ bool commit() {
    for (;;) {
      const int tag = fr.tag;
      const unsigned open = ~__ballot_sync(FULL, tag >= 0);
      if (open & 1u) return true;
      if (fr.short_of_room()) {
        fr.compact();
        if (fr.near == 0) return false;  // (nothing is left of the front, hence of the far keys)
        continue;
      }
      if (fr.done >= fr.ef && !fr.among_closest(shfl64(fr.front, 0))) return false;
      // lane i: what nodes 0 .. i bring, its smallest image and its number
      unsigned least = tag >= 0 ? lds32(board + Board::kLeast + 4 * (tag & (kBuffers - 1))) : ~0u;
      int count = tag >= 0 ? tag >> kCountAt : 0;
#pragma unroll
      for (int o = 1; o < kBuffers; o *= 2) {
        const unsigned l = __shfl_up_sync(FULL, least, o);
        const int c = __shfl_up_sync(FULL, count, o);
        if (lane >= o) {
          least = min(least, l);
          count += c;
        }
      }
      const unsigned before = __shfl_up_sync(FULL, least, 1);
      const bool too = lane == 0 || (lane < kMost && tag >= 0 && (unsigned)(fr.front >> 32) < before &&
                                     fr.done + lane < fr.ef && fr.done + fr.far + lane + 1 + count <= fr.cap);
      const int r = __ffs(~__ballot_sync(FULL, too)) - 1;  // (at most kMost)
      const int total = __shfl_sync(FULL, count, r - 1);
      fr.pop_some(r);
      wc.expansions += r;
      for (int base = 0; base < total; base += 32) {
        if (base > 0 && fr.short_of_room()) fr.compact();
        const int g = min(base + lane, total - 1);
        int i = 0;
        for (int j = 0; j + 1 < r; ++j) i += __shfl_sync(FULL, count, j) <= g ? 1 : 0;
        const int first = __shfl_sync(FULL, count, (i - 1) & 31);
        const unsigned place = place_of(__shfl_sync(FULL, tag, i) & (kBuffers - 1));
        take_in(lds64(place + 8 * (g - (i > 0 ? first : 0))), base + lane < total, r > 1);
      }
    }
  }

  // From the frontier's first keys to the end of the walk: expanded keys and expansions are those of the literal walk.
  __device__ __forceinline__ void run() {
    for (;;) {
      if (fr.near < P && fr.far > 0) fr.refill();
      if (fr.near == 0) return;
      prepare();  // the first key among others: a commit ends in front of one that is not prepared
      if (!commit()) return;
    }
  }
};

}  // namespace hnsw
