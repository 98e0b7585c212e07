// The graph walk of one CTA per query, which prepares several nodes at a time.
//
// The ef-bounded best-first search of one layer is a chain: expand the closest unexpanded node, merge what its
// neighbours are worth, look again.  Run literally (beam_layer in beam.cuh), every link of that chain costs an
// adjacency row, a gather of vectors and a list merge, one after the other: about 3600 cycles, of which the
// memory latencies are most, and nothing of one link overlaps with the next.
//
// But the nodes that will be expanded next are known: nearly every key that sits among the first few unexpanded
// keys of the list is expanded sooner or later (counted on four of the benchmark's graphs: preparing the first
// eight at a time prepares 1.00 to 1.08 nodes and evaluates 1.05 to 1.25 rows for each one the literal walk does).
// So a ROUND
//   selects   up to P unexpanded keys in list order that are not prepared yet,
//   prepares  them together: adjacency rows, visited filter, distances of all their new neighbours, kept in a
//             buffer per node, and
//   commits   prepared nodes in exactly the order of the literal walk: the closest unexpanded key, as long as it
//             is a prepared one.
// Nothing a prepared node brings is seen by the list or the visited table before its commit, so list, visited
// nodes and results are those of the literal walk, step for step.  A round commits 3.2 nodes on average with P = 4,
// 4.7 with P = 8, so the two memory round trips are paid once for that many expansions instead of for each, and there is
// enough to evaluate for the W warps of a CTA.  Warp 0 owns the list and the commits; all share the preparation.
//
// With fewer queries than the chip has warp slots this shortens the chain that a launch waits for; with more it loses to
// one warp per query, whose helpers never wait (the rules that choose are in search_walk.cuh).
#pragma once
#include "beam.cuh"

namespace hnsw {

// The candidate/result list: ascending keys (distance image, 2 * id + taken) in shared memory, capacity ef.  With the
// flag in the lowest bit keys compare as they stand.  A group of up to 32 keys is merged at once: places by binary
// search (the same number of steps in every lane), ranks among the group, then one bit per place of the new list
// says whether it holds a newcomer; the old key of a place is the one that many places further down, so that the list
// moves 32 keys at a time whatever the group's size.
struct KeyList {
  unsigned keys;   // shared-memory address of cap + 1 keys; those from `size` on read ~0
  unsigned marks;  // a bit per place
  unsigned spot;   // 32 words of scratch
  int cap, size;
  int cursor;      // every key before it is taken
  uint2 worst;     // the ef-th key (~0 while there is room)
  int lane;
  unsigned lower;  // lanes below this one

  __host__ __device__ static int bytes(int cap) { return (cap + 2) / 2 * 16 + (cap + 127) / 128 * 16 + 128; }
  __device__ __forceinline__ void bind(unsigned smem, int cap_) {
    keys = smem;
    cap = cap_;
    marks = keys + (cap + 2) / 2 * 16;
    spot = marks + (cap + 127) / 128 * 16;
    lane = lane_number();
    lower = (1u << lane) - 1u;
  }
  static __device__ __forceinline__ bool less(uint2 a, uint2 b) {
    return ((unsigned long long)a.x << 32 | a.y) < ((unsigned long long)b.x << 32 | b.y);
  }
  // list = {(image, id)}
  __device__ __forceinline__ void seed(unsigned image, unsigned id) {
    for (int i = lane; i < (cap + 2) / 2; i += 32) sts128(keys + 16 * i, ~0u, ~0u, ~0u, ~0u);
    __syncwarp();
    if (lane == 0) sts64(keys, image, 2 * id);
    size = 1;
    cursor = 0;
    __syncwarp();
    load_worst();
  }

  // Merges the g <= 32 keys at `group` (overwritten up to the next multiple of four), keeping the ef smallest; keys
  // that are listed already or come twice enter once.
  __device__ __forceinline__ void merge(unsigned group, int g) {
    const uint2 key = lane < g ? lds64(group + 8 * lane) : make_uint2(~0u, ~0u);
    bool keep = less(key, worst);
    if (!__any_sync(FULL, keep)) return;
    // at: address of the first key that is not below the new one.  Steps past the end read the last place, ~0.
    unsigned at = keys;
    const unsigned end = keys + 8 * cap;
    if (size > 255) {
      int step = 256;
      while (2 * step <= size) step *= 2;
      for (; step > 128; step >>= 1)
        if (less(lds64(min(at + 8 * step - 8, end)), key)) at += 8 * step;
    }
    // four ways at a time: three reads under way together, four dependent steps instead of eight
#pragma unroll
    for (int step = 64; step > 0; step >>= 2) {
      int n = 0;
#pragma unroll
      for (int u = 1; u <= 3; ++u) n += less(lds64(min(at + 8 * u * step - 8, end)), key) ? 1 : 0;
      at += 8 * n * step;
    }
    {
      const uint2 v = lds64(at);
      keep = keep && !(v.x == key.x && (v.y | 1u) == key.y + 1u);  // listed already?
    }
    if (!keep && lane < ((g + 3) & ~3)) sts64(group + 8 * lane, ~0u, ~0u);
    for (int i = lane; i < (cap + 31) / 32; i += 32) sts32(marks + 4 * i, 0u);
    __syncwarp();
    int rank = 0;  // among the newcomers
    for (int j = 0; j < g; j += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) rank += less(lds64(group + 8 * (j + u)), key) ? 1 : 0;
    }
    // equal keys have equal ranks: one of them stays
    if (keep) sts32(spot + 4 * rank, lane);
    __syncwarp();
    const bool twice = keep && lds32(spot + 4 * (rank & 31)) != (unsigned)lane;
    if (__any_sync(FULL, twice)) {
      keep = keep && !twice;
      rank = 0;
      for (unsigned m = __ballot_sync(FULL, keep); m; m &= m - 1) {
        const int b = __ffs(m) - 1;
        const uint2 other = make_uint2(__shfl_sync(FULL, key.x, b), __shfl_sync(FULL, key.y, b));
        rank += less(other, key) ? 1 : 0;
      }
    }
    const int place = (int)((at - keys) >> 3) + rank;
    const bool in = keep && place < cap;
    if (in) atomic_or_shared(marks + 4 * (place >> 5), 1u << (place & 31));
    int below = __popc(__ballot_sync(FULL, in));  // newcomers in the windows not yet moved
    if (below == 0) return;
    const int grown = min(cap, size + __popc(__ballot_sync(FULL, keep)));
    const int first = (int)__reduce_min_sync(FULL, in ? (unsigned)place : 0x7fffffffu);
    __syncwarp();
    const unsigned bit = 1u << lane;
    const int lowest = first >> 5;
    int w = (grown - 1) >> 5;
    // four windows at a time, top down: all are read before the first is written, and what they read lies below
    // everything the windows before them wrote
    for (; w >= lowest; w -= 4) {
      unsigned word[4];
      uint2 v[4];
      bool moves[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) word[u] = lds32(marks + 4 * max(w - u, 0));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = 32 * (w - u) + lane;
        below -= __popc(word[u]);
        moves[u] = w - u >= lowest && i < grown && !(word[u] & bit);
        v[u] = lds64(moves[u] ? keys + 8 * (i - below - __popc(word[u] & lower)) : keys);
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (moves[u]) sts64(keys + 8 * (32 * (w - u) + lane), v[u].x, v[u].y);
      __syncwarp();
    }
    __syncwarp();
    if (in) sts64(keys + 8 * place, key.x, key.y);
    size = grown;
    cursor = min(cursor, first);
    __syncwarp();
    load_worst();
  }
  __device__ __forceinline__ void load_worst() {
    const uint2 k = lds64(keys + 8 * (cap - 1));
    worst = make_uint2(__shfl_sync(FULL, k.x, 0), __shfl_sync(FULL, k.y, 0));
  }

  // Takes the first `want` keys that are not taken, in order: copies go to the places req[0 .. want - 1], and of the one
  // after them to req[want].  Returns how many were copied.
  __device__ __forceinline__ int take(int want, unsigned req) {
    int have = 0;
    for (int c = cursor;; c += 32) {
      const int i = c + lane;
      uint2 v = make_uint2(0u, 1u);
      if (i < size) v = lds64(keys + 8 * i);
      const bool open = !(v.y & 1u);
      const unsigned m = __ballot_sync(FULL, open);
      const int r = have + __popc(m & lower);
      if (open && r <= want) sts64(req + 8 * r, v.x, v.y);
      if (open && r < want) sts32(keys + 8 * i + 4, v.y | 1u);
      have += __popc(m);
      if (have > want) {
        cursor = c + __ffs(__ballot_sync(FULL, open && r == want)) - 1;
        break;
      }
      if (c + 32 >= size) {
        cursor = size;
        break;
      }
    }
    __syncwarp();
    return min(have, want + 1);
  }
};

// What the warps of one walk tell each other, in shared memory: 32-bit words at these offsets.
template <int P>
struct WalkBoard {
  static constexpr int kOp = 0, kNodes = 4, kPool = 8, kQuery = 12;  // operation, nodes of the round, rows in the pool, query
  static constexpr int kNode = 16;                // P node ids
  static constexpr int kPlace = kNode + 4 * P;    // and the addresses of the buffers their neighbours go to
  static constexpr int kCount = kPlace + 4 * P;   // new neighbours of each
  static constexpr int kReq = kCount + 4 * P;     // P + 1 selected keys
  static constexpr int kBytes = (kReq + 8 * (P + 1) + 15) / 16 * 16;
};
// (the last two in frontier_walk.cuh only)
enum { kWalkOver = 0, kWalkQuery = 1, kWalkRound = 2, kWalkRows = 3, kWalkNode = 4, kWalkKeys = 5 };

template <class Dist, int W, int P>
struct Walk {
  static constexpr int kBuffers = 2 * P;
  static_assert(W > 1 && kBuffers <= 32, "a lane stands for a buffer");
  using Board = WalkBoard<P>;

  Dist de;
  KeyList list;
  VisitedPairs vis;
  unsigned found;  // shared-memory address of kBuffers x stride keys: the prepared nodes' new neighbours
  unsigned pool;   // of the rows to evaluate: (id, address of the key's place in `found`)
  unsigned board;
  const int* rows;  // adjacency table of layer 0
  int stride;       // ints per adjacency row (= keys per buffer)
  int lane;
  WalkCounters wc;

  // shared memory of one walk, without the distance engine's own
  __host__ __device__ static size_t smem_bytes(int ef, int stride, int ventries, long long n) {
    return (size_t)KeyList::bytes(ef) + (size_t)kBuffers * stride * 8 + (size_t)P * stride * 8 + Board::kBytes +
           VisitedPairs::smem_bytes(ventries, n);
  }
  __device__ __forceinline__ void bind(unsigned char* smem, int ef, int stride_, int ventries, long long n) {
    unsigned at = kept(smem_addr(smem));
    list.bind(at, ef);
    found = at += KeyList::bytes(ef);
    pool = at += kBuffers * stride_ * 8;
    board = at += P * stride_ * 8;
    vis.bind_table(at + Board::kBytes, ventries, n);
    stride = stride_;
    lane = lane_number();
    wc = WalkCounters{0, 0, 0, 0};
  }
  static __device__ __forceinline__ int warp() { return __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0); }
  __device__ __forceinline__ unsigned place_of(int buffer) const { return found + 8 * stride * buffer; }
  // a word of the board, known to be the same in every lane
  __device__ __forceinline__ int posted(int at) const { return __shfl_sync(FULL, (int)lds32(board + at), 0); }
  __device__ __forceinline__ const int* row_of(int id) const {
    return rows + (size_t)id * stride;
  }

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
      const bool slot = base + lane < stride;
      const int l = slot ? base + lane : 0;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i < count) nid[i] = __ldg(row_of(node[i]) + l);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (i < count) {
          const bool known = vis.knows(nid[i]);
          const bool fresh = slot && nid[i] >= 0 && !known;
          const unsigned m = __ballot_sync(FULL, fresh);
          const int before = __popc(m & list.lower);
          int at = 0;
          if (lane == 0) at = (int)atomic_add_shared(board + Board::kPool, __popc(m));
          at = __shfl_sync(FULL, at, 0);
          if (fresh) sts64(pool + 8 * (at + before), (unsigned)nid[i], place[i] + 8 * (have[i] + before));
          have[i] += __popc(m);
        }
      }
    }
  }
  // this warp's share of the round on the board
  __device__ __forceinline__ void filter_posted(int w) {
    constexpr int N = (P + W - 1) / W;
    const int nsel = posted(Board::kNodes);
    if (w >= nsel) return;
    const int count = (nsel - w + W - 1) / W;
    int node[N], have[N];
    unsigned place[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int c = min(w + W * i, P - 1);
      node[i] = posted(Board::kNode + 4 * c);
      place[i] = (unsigned)posted(Board::kPlace + 4 * c);
    }
    filter_rows(node, place, count, have);
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < count && lane == 0) sts32(board + Board::kCount + 4 * (w + W * i), (unsigned)have[i]);
  }

  // Warps 1 .. W - 1: every operation starts and ends at a block barrier, as warp 0's do.
  __device__ __forceinline__ void help(const float* queries) {
    const int w = warp();
    for (;;) {
      __syncthreads();
      const int op = posted(Board::kOp);
      if (op == kWalkOver) return;
      if (op == kWalkQuery) {
        if (!Dist::kSharedQuery) load(queries);
        vis.clear(w, W);
      } else {
        if (op == kWalkRound) {
          filter_posted(w);
          __syncthreads();
        }
        de.template eval_pool<false>(pool, posted(Board::kPool), w, W, 0);
      }
      __syncthreads();
    }
  }
  // the query whose number is on the board
  __device__ __forceinline__ void load(const float* queries) {
    de.load_query(queries + (size_t)(unsigned)posted(Board::kQuery) * de.t.d);
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
    de.template eval_pool<false>(pool, n, 0, W, 0);
    __syncthreads();
    wc.evals += n;
  }
  // query `i` of `queries`
  __device__ __forceinline__ void start(const float* queries, long long i) {
    if (lane == 0) sts32(board + Board::kQuery, (unsigned)i);
    post(kWalkQuery);
    load(queries);
    vis.clear(0, W);
    __syncthreads();
  }
  __device__ __forceinline__ void finish() { post(kWalkOver); }

  // Greedy walk through layers top .. 1 (same rule as greedy_descent in beam.cuh).
  __device__ __forceinline__ void descend(const GraphView& g, int& cur, float& dcur) {
    cur = g.enter_point;
    if (lane == 0) sts64(pool, (unsigned)cur, found);
    evaluate_rows(1);
    dcur = ord2f(__shfl_sync(FULL, lds32(found), 0));  // (the shuffle tells the compiler that all lanes agree)
    for (int l = g.max_level; l > 0; --l) {
      for (;;) {
        const int* row = g.rowsU + ((size_t)__ldg(g.upper_base + cur) + (l - 1)) * g.strideU;
        wc.sweeps += 1;
        int n = 0;
        for (int base = 0; base < g.strideU; base += 32) {
          const int li = base + lane;
          const int nid = li < g.strideU ? __ldg(row + li) : -1;
          const unsigned m = __ballot_sync(FULL, nid >= 0);
          const int at = n + __popc(m & list.lower);
          if (nid >= 0) sts64(pool + 8 * at, (unsigned)nid, found + 8 * at);
          n += __popc(m);
        }
        if (n == 0) break;
        evaluate_rows(n);
        int best_id = cur;
        float best_d = dcur;
        for (int base = 0; base < n; base += 32) {
          uint2 k = base + lane < n ? lds64(found + 8 * (base + lane)) : make_uint2(~0u, ~0u);
          if (k.x < f2ord(-__int_as_float(0x7f800000))) k.x = ~0u;  // a negative NaN is not closest
          const unsigned least = __reduce_min_sync(FULL, k.x);
          const int at = __ffs(__ballot_sync(FULL, k.x == least)) - 1;  // first in row order
          const int id = __shfl_sync(FULL, (int)k.y, at);
          if (ord2f(least) < best_d) {
            best_d = ord2f(least);
            best_id = id;
          }
        }
        __syncwarp();
        if (best_id == cur) break;
        cur = best_id;
        dcur = best_d;
      }
    }
  }

  __device__ __forceinline__ void seed(int id, float dist) {
    list.seed(f2ord(dist), (unsigned)id);
    if (lane == 0) vis.test_and_set(id);
    __syncwarp();
  }

  // The n neighbours at `place` enter the visited table; those the table did not know and that may enter the list go to
  // the queue in the pool's memory, and the smallest distance image among this lane's to `least`.
  __device__ __forceinline__ int append(unsigned place, int n, int queued, unsigned& least) {
    for (int base = 0;;) {
      const bool have = base + lane < n;
      const uint2 key = lds64(have ? place + 8 * (base + lane) : place);
      const bool known = vis.test_and_set((int)key.y, have);
      const bool in = have && !known && key.x <= list.worst.x;
      const unsigned m = __ballot_sync(FULL, in);
      if (in) sts64(pool + 8 * (queued + __popc(m & list.lower)), key.x, 2 * key.y);
      if (in) least = min(least, key.x);
      queued += __popc(m);
      base += 32;
      if (base >= stride) return queued;
    }
  }

  // The prepared nodes, in list order: lane r < c has the r-th one's key (distance image, id), the buffer
  // with its new neighbours and their number.
  struct Prepared {
    unsigned image, node;
    int buffer, count;
  };

  // Commits the first of the c prepared nodes and those after it as long as each is the closest unexpanded one when its
  // turn comes: closer than `next`, the closest key that is neither prepared nor expanded, and than every neighbour
  // the nodes before it bring.  (A node's rank in the list does not change while nothing closer comes in, so all of
  // them are in the list if they are now.)  The neighbours of the committed nodes then enter the list as one group:
  // what it ends with does not depend on their order.  Returns how many were committed, 0 when the walk is over: the
  // closest unexpanded key has left the list.
  __device__ __forceinline__ int commit(const Prepared& mine, int c, unsigned next) {
    unsigned image = __shfl_sync(FULL, mine.image, 0);
    if (KeyList::less(list.worst, make_uint2(image, 2 * __shfl_sync(FULL, mine.node, 0)))) return 0;
    unsigned least = ~0u;
    int queued = 0, done = 0;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if (r > 0) {
        // (equal distances wait for their turn at the front, where the whole keys are compared)
        image = __shfl_sync(FULL, mine.image, r);
        if (r >= c || image >= next || image >= list.worst.x) break;
        if (__any_sync(FULL, least <= image)) break;
      }
      queued = append(place_of(__shfl_sync(FULL, mine.buffer, r)), __shfl_sync(FULL, mine.count, r), queued, least);
      ++done;
    }
    wc.expansions += done;
    wc.inserts += queued;
    __syncwarp();
    for (int base = 0; base < queued; base += 32) list.merge(pool + 8 * base, min(32, queued - base));
    __syncwarp();
    return done;
  }

  // From the list's seeds to its end: on return the list holds what the literal best-first walk ends with.
  __device__ __forceinline__ void run() {
    Prepared mine{~0u, ~0u, 0, 0};
    int c = 0;
    for (;;) {
      // nodes whose key has left the list: the last ones
      c = __popc(__ballot_sync(FULL, lane < c && !KeyList::less(list.worst, make_uint2(mine.image, 2 * mine.node))));
      // select.  At least one buffer is free: every round commits the first key of those selected so far.
      const int want = min(P, kBuffers - c);
      const int copied = list.take(want, board + Board::kReq);
      const int nsel = min(want, copied);
      unsigned next = ~0u;  // distance image of the closest key that is neither prepared nor expanded
      if (copied > nsel) next = __shfl_sync(FULL, lds32(board + Board::kReq + 8 * nsel), 0);
      if (nsel > 0) {
        // the nodes selected take the lanes c .. c + nsel - 1 and free buffers
        int b = lane - c;
        if (c > 0) {
          const unsigned used = __reduce_or_sync(FULL, lane < c ? 1u << mine.buffer : 0u);
          if (lane < kBuffers && !((used >> lane) & 1u)) sts32(list.spot + 4 * __popc(~used & list.lower), lane);
          __syncwarp();
          b = (int)lds32(list.spot + 4 * (b & (kBuffers - 1)));
        }
        const bool chosen = lane >= c && lane < c + nsel;
        if (chosen) {
          const uint2 k = lds64(board + Board::kReq + 8 * (lane - c));
          mine.image = k.x;
          mine.node = k.y >> 1;
          mine.buffer = b;
        }
        if (chosen) {
          sts32(board + Board::kNode + 4 * (lane - c), mine.node);
          sts32(board + Board::kPlace + 4 * (lane - c), place_of(mine.buffer));
        }
        if (lane == 0) {
          sts32(board + Board::kNodes, nsel);
          sts32(board + Board::kPool, 0);
        }
        post(kWalkRound);
        filter_posted(0);
        __syncthreads();
        const int total = posted(Board::kPool);
        de.template eval_pool<false>(pool, total, 0, W, 0);
        __syncthreads();
        if (chosen) mine.count = (int)lds32(board + Board::kCount + 4 * (lane - c));
        wc.evals += total;
        const int before = c;
        c += nsel;
        if (before > 0) {
          // bring old and new nodes into list order
          const uint2 k = make_uint2(mine.image, mine.node);
          int rank = 0;
#pragma unroll
          for (int i = 0; i < kBuffers; ++i) {
            const uint2 o = make_uint2(__shfl_sync(FULL, k.x, i), __shfl_sync(FULL, k.y, i));
            rank += (i < c && KeyList::less(o, k)) ? 1 : 0;
          }
          if (lane < c) sts128(pool + 16 * rank, mine.image, mine.node, mine.buffer, mine.count);
          __syncwarp();
          if (lane < c) {
            const uint2 lo = lds64(pool + 16 * lane), hi = lds64(pool + 16 * lane + 8);
            mine = Prepared{lo.x, lo.y, (int)hi.x, (int)hi.y};
          }
          __syncwarp();
        }
      }
      if (c == 0) break;
      const int done = commit(mine, c, next);
      if (done == 0) break;
      c -= done;
      mine.image = __shfl_down_sync(FULL, mine.image, done);
      mine.node = __shfl_down_sync(FULL, mine.node, done);
      mine.buffer = __shfl_down_sync(FULL, mine.buffer, done);
      mine.count = __shfl_down_sync(FULL, mine.count, done);
    }
  }
};

}  // namespace hnsw
