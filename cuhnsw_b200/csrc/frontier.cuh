// What the ef-bounded best-first walk of one CTA has to remember (frontier_walk.cuh), without a list of the ef closest keys in order.
//
// The literal walk keeps the ef closest keys seen so far sorted, expands the closest one that is not expanded yet and ends
// when all are.  Little of that order is needed:
//   - the next nodes are the smallest keys that are not expanded, so only the smallest few of those have to be in order;
//   - a key is among the ef closest if fewer than ef keys that were seen are smaller.  All keys smaller than the
//     smallest unexpanded one are expanded, so that key is listed exactly if fewer than ef EXPANDED keys are smaller,
//     which nobody has to count before ef keys are expanded; and once it is not listed, none is, and the walk is over;
//   - the ef closest keys at the end are the ef smallest expanded ones.
// So the keys live in three places: the FRONT, up to 32 of the smallest unexpanded keys, sorted, one per lane in
// registers; the FAR keys, all other unexpanded ones, in no order; and the expanded keys (DONE), in the order of their
// expansion.  Far and done share one array of slots in shared memory and grow towards each other.  A newcomer that does
// not belong to the front costs one store.  When the front runs short, 10 or more keys are picked from the far ones
// (by bisection on the key); when the slots run out, the ef smallest keys are kept and the largest of them becomes the
// limit that newcomers have to beat, which the literal walk's worst key is at all times.  Counted at ef 200 (120 000 x 50), per
// expansion: 0.66 keys into the front, 0.03 refills, 0.01 times the slots run out.
//
// Every key must be there once, or it would be expanded twice and counted twice.  The visited table forgets ids, so a
// newcomer whose bucket is full - only those can have been forgotten - is looked up among the keys (one expansion in 14).
//
// Bound: latency of one warp's dependent shared-memory reads, shuffles and ballots.  For one warp per query it was no gain
// over the sorted list of WarpList (298 against 315 instructions per expansion, 10 000 queries 1.59 against 1.36 ms).
#pragma once
#include "beam.cuh"

namespace hnsw {

struct Frontier : VisitedTable {
  static constexpr unsigned long long kNone = ~0ull;  // above every key
  static constexpr int kSlack = 16;                   // keys kept beyond ef when the slots run out: at most this many
  static constexpr int kChunk = 32;                   // newcomers that come at once
  static constexpr int kMinSlots = kChunk + 1 + kSlack + 15;

  int lane;
  unsigned lower;    // lanes below this one
  unsigned slots;    // shared-memory address of `cap` keys
  unsigned scratch;  // of 32 keys
  int cap, ef;
  int done;  // expanded keys: slots 0 .. done - 1
  int far;   // slots cap - far .. cap - 1
  int near;  // keys in the front
  unsigned long long front;  // lane l: the l-th smallest unexpanded key
  unsigned long long split;  // far keys are not below it, front keys are
  unsigned long long limit;  // a key that is not below it is not among the ef closest
  unsigned step;             // image distance that the last refill went up by
  int tag;                   // goes where the lane's front key goes; -1 for a key that comes in, and without a key

  // slots of a walk that keeps ef keys: what it needs at least, and twice the usual number of newcomers of a round more
  __host__ __device__ static int slots_for(int ef) { return least_slots(ef) + 64; }
  __host__ __device__ static int least_slots(int ef) { return (ef + kMinSlots + 1) / 2 * 2; }
  __host__ __device__ static size_t smem_bytes(int cap) { return (size_t)cap * 8 + kChunk * 8; }
  __device__ __forceinline__ void bind(unsigned smem, int ef_, int cap_, int entries, long long n) {
    lane = lane_number();
    lower = (1u << lane) - 1u;
    slots = kept(smem);
    ef = ef_;
    cap = cap_;
    scratch = slots + 8 * cap;
    bind_table(scratch + kChunk * 8, entries, n);
  }
  // nothing seen yet (the visited table is cleared by its owner)
  __device__ __forceinline__ void reset() {
    done = far = near = 0;
    front = split = limit = kNone;
    step = 1u << 18;
    tag = -1;
  }
  static __device__ __forceinline__ unsigned long long word(uint2 v) { return ((unsigned long long)v.y << 32) | v.x; }
  __device__ __forceinline__ unsigned long long slot(int i) const { return key_at(slots, i); }
  __device__ __forceinline__ void set_slot(int i, unsigned long long k) const {
    sts64(slots + 8 * i, (unsigned)k, (unsigned)(k >> 32));
  }
  // room for one more expansion and the newcomers of one chunk of its neighbours
  __device__ __forceinline__ bool short_of_room() const { return done + far + kChunk + 1 > cap; }

  // ---- counting and bisection ----

  // (Slots are read four windows of 32 at a time, so that their reads are under way together.)
  // Keys below t among the `count` slots from `first` on: this lane's share.
  __device__ __forceinline__ int share_below(int first, int count, unsigned long long t) const {
    int c = 0;
    for (int base = 0; base < count; base += 128) {
      unsigned long long k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = slot(first + min(base + 32 * u + lane, count - 1));
#pragma unroll
      for (int u = 0; u < 4; ++u) c += base + 32 * u + lane < count && k[u] < t ? 1 : 0;
    }
    return c;
  }
  __device__ __forceinline__ int below(int first, int count, unsigned long long t) const {
    return __reduce_add_sync(FULL, share_below(first, count, t));
  }
  // A bound that `want` to `room` of the slots' keys lie below (want < count; keys are different): searched upwards from
  // `lo`, which none of them lies below, in steps that start at `step`.
  __device__ __forceinline__ unsigned long long bound(int first, int count, int want, int room, unsigned long long lo) {
    const unsigned long long from = lo;
    unsigned long long hi = kNone, at = lo + ((unsigned long long)step << 32);
    unsigned stride = step;
    bool bounded = false;
    if (at < lo) at = kNone;
    for (;;) {
      const int c = below(first, count, at);
      if (c > room) {
        hi = at;
        bounded = true;
      } else if (c < want) {
        lo = at;
      } else {
        break;
      }
      if (!bounded) {
        stride = stride < (1u << 29) ? 4 * stride : stride;
        at = lo + ((unsigned long long)stride << 32);
        if (at < lo) at = kNone;  // all of them lie below it
      } else {
        if (hi - lo < 2) break;  // (two equal keys: not reached)
        at = lo + (hi - lo) / 2;
      }
    }
    step = max(1u << 10, (unsigned)((at - from) >> 32));
    return at;
  }
  // The n <= 32 keys in `scratch` in ascending order; lane l returns the l-th.
  __device__ __forceinline__ unsigned long long sorted_scratch(int n) const {
    if (lane >= n) sts64(scratch + 8 * lane, ~0u, ~0u);
    __syncwarp();
    const unsigned long long mine = word(lds64(scratch + 8 * lane));
    int rank = 0;
    for (int j = 0; j < n; j += 4) {
      uint4 v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) v[u] = lds128(scratch + 8 * j + 16 * u);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        rank += word(make_uint2(v[u].x, v[u].y)) < mine ? 1 : 0;
        rank += word(make_uint2(v[u].z, v[u].w)) < mine ? 1 : 0;
      }
    }
    __syncwarp();
    if (lane < n) sts64(scratch + 8 * rank, (unsigned)mine, (unsigned)(mine >> 32));
    __syncwarp();
    return word(lds64(scratch + 8 * lane));
  }
  // Those of the first `count` slots (kDown: of the last, from the end) whose keys are below t move together in place;
  // returns their number.  What is read lies at or behind everything written.
  template <bool kDown>
  __device__ __forceinline__ int keep_below(int count, unsigned long long t) const {
    int n = 0;
    for (int base = 0; base < count; base += 128) {
      unsigned long long k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = min(base + 32 * u + lane, count - 1);
        k[u] = slot(kDown ? cap - 1 - i : i);
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool stay = base + 32 * u + lane < count && k[u] < t;
        const unsigned m = __ballot_sync(FULL, stay);
        const int at = n + __popc(m & lower);
        if (stay) set_slot(kDown ? cap - 1 - at : at, k[u]);
        n += __popc(m);
      }
      __syncwarp();
    }
    return n;
  }

  // ---- keys coming and going ----

  // Is this key here already?  (the same in every lane)
  __device__ __forceinline__ bool listed(unsigned long long k) const {
    const unsigned id = (unsigned)k;
    bool hit = front == k;
    for (int base = 0; base < done; base += 64) {
      const int i = base + 2 * lane;
      const uint4 v = lds128(slots + 8 * min(i, cap - 2));
      hit = hit || (i < done && v.x == id) || (i + 1 < done && v.z == id);
    }
    if (k >= split) {
      for (int base = 0; base < far; base += 64) {
        const int i = base + 2 * lane;  // counted from the last slot
        const uint4 v = lds128(slots + 8 * max(cap - 2 - i, 0));
        hit = hit || (i < far && v.z == id) || (i + 1 < far && v.x == id);
      }
    }
    return __any_sync(FULL, hit);
  }
  __device__ __forceinline__ void push_far(unsigned long long k) {
    if (lane == 0) set_slot(cap - 1 - far, k);
    ++far;
  }
  // One key (the same in every lane) that was below `split` when its chunk came takes its place in the front: lane l has
  // the smaller of its key and what comes up to it, the larger of the new key and the one below.
  __device__ __forceinline__ void push_front(unsigned long long k) {
    if (near == 32) {
      const unsigned long long out = max(shfl64(front, 31), k);
      push_far(out);
      split = min(split, out);  // (a key of the same chunk may have taken it below k)
    } else {
      ++near;
    }
    const unsigned lo = __shfl_up_sync(FULL, (unsigned)front, 1), hi = __shfl_up_sync(FULL, (unsigned)(front >> 32), 1);
    const unsigned long long before = lane > 0 ? ((unsigned long long)hi << 32) | lo : 0ull;
    const int t = __shfl_up_sync(FULL, tag, 1);
    tag = front < k ? tag : before < k ? -1 : t;
    front = min(front, max(before, k));
  }
  // Up to 32 newcomers, one per lane.  `suspect`: the visited table may have forgotten this one.  The caller has seen to
  // it that there is room.
  __device__ __forceinline__ void take(unsigned long long k, bool active, bool suspect, WalkCounters& wc) {
    bool in = active && k < limit;
    for (unsigned m = __ballot_sync(FULL, in && suspect); m; m &= m - 1) {
      const int b = __ffs(m) - 1;
      if (listed(shfl64(k, b)) && lane == b) in = false;
    }
    const unsigned im = __ballot_sync(FULL, in);
    const bool away = in && k >= split;
    const unsigned fm = __ballot_sync(FULL, away);
    if (away) set_slot(cap - 1 - far - __popc(fm & lower), k);
    far += __popc(fm);
    wc.inserts += __popc(im);
    for (unsigned m = im & ~fm; m; m &= m - 1) push_front(shfl64(k, __ffs(m) - 1));
    __syncwarp();
  }
  // the r smallest unexpanded keys leave the front for the expanded ones
  __device__ __forceinline__ void pop_some(int r) {
    if (lane < r) set_slot(done + lane, front);
    const unsigned lo = __shfl_down_sync(FULL, (unsigned)front, r), hi = __shfl_down_sync(FULL, (unsigned)(front >> 32), r);
    front = lane < 32 - r ? ((unsigned long long)hi << 32) | lo : kNone;
    const int t = __shfl_down_sync(FULL, tag, r);
    tag = lane < 32 - r ? t : -1;
    near -= r;
    done += r;
  }
  // Is key k, smaller than every unexpanded one but itself, among the ef closest?
  __device__ __forceinline__ bool among_closest(unsigned long long k) const {
    return done < ef || below(0, done, k) < ef;
  }

  // The smallest far keys join the front: 10 or more if there are as many, up to what fits.
  __device__ __forceinline__ void refill() {
    const int room = 32 - near;
    __syncwarp();
    int m = 0;
    if (far <= room) {
      if (lane < far) {
        const uint2 v = lds64(slots + 8 * (cap - 1 - lane));
        sts64(scratch + 8 * lane, v.x, v.y);
      }
      m = far;
      far = 0;
      split = kNone;
    } else {
      const unsigned long long t = bound(cap - far, far, min(10, room), room, split);
      int kept_keys = 0;
      for (int base = 0; base < far; base += 64) {
        unsigned long long k[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) k[u] = slot(cap - 1 - min(base + 32 * u + lane, far - 1));
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const bool have = base + 32 * u + lane < far, out = have && k[u] < t, stay = have && k[u] >= t;
          const unsigned om = __ballot_sync(FULL, out), sm = __ballot_sync(FULL, stay);
          const int at = m + __popc(om & lower);
          if (out && at < room) sts64(scratch + 8 * at, (unsigned)k[u], (unsigned)(k[u] >> 32));
          if (stay) set_slot(cap - 1 - kept_keys - __popc(sm & lower), k[u]);
          m += __popc(om);
          kept_keys += __popc(sm);
        }
        __syncwarp();
      }
      far = kept_keys;
      split = t;
      m = min(m, room);
    }
    const unsigned long long k = sorted_scratch(m);
    const unsigned lo = __shfl_sync(FULL, (unsigned)k, (lane - near) & 31);
    const unsigned hi = __shfl_sync(FULL, (unsigned)(k >> 32), (lane - near) & 31);
    if (lane >= near && lane < near + m) front = ((unsigned long long)hi << 32) | lo;
    near += m;
  }

  // The slots have run out: the ef smallest keys stay (and up to kSlack more), the others cannot be among the ef closest.
  __device__ __forceinline__ void compact() {
    __syncwarp();
    int total = done + far + near;
    unsigned long long lo = 0, hi = limit;
    if (hi == kNone) {  // no limit yet: from above the largest key down
      unsigned top = near > 0 && front != kNone ? (unsigned)(front >> 32) : 0u;
      for (int base = 0; base < done + far; base += 32) {
        const int i = min(base + lane, done + far - 1);
        top = max(top, lds64(slots + 8 * (i < done ? i : cap - far + (i - done))).y);
      }
      top = __reduce_max_sync(FULL, top);
      if (top != ~0u) hi = (unsigned long long)(top + 1) << 32;
    }
    if (done < ef && near > 0) lo = shfl64(front, 0);  // only expanded keys lie below it
    while (total > ef + kSlack && hi - lo > 1) {
      const unsigned long long mid = lo + (hi - lo) / 2;
      const int c = __reduce_add_sync(
          FULL, (front < mid ? 1 : 0) + share_below(0, done, mid) + share_below(cap - far, far, mid));
      if (c >= ef) {
        hi = mid;
        total = c;
      } else {
        lo = mid;
      }
    }
    limit = hi;
    done = min(keep_below<false>(done, hi), cap - kChunk - 1);
    far = min(keep_below<true>(far, hi), cap - kChunk - 1 - done);
    if (front >= hi) {
      front = kNone;
      tag = -1;
    }
    near = __popc(__ballot_sync(FULL, front != kNone));
    if (far == 0) split = kNone;
  }

  // ---- what the walk found: the expanded keys ----

  // The m <= 32 smallest (all of them if there are fewer); lane l returns the l-th, kNone past the last.
  __device__ __forceinline__ unsigned long long closest(int m) {
    __syncwarp();
    unsigned long long t = kNone;
    if (done > 32) {
      unsigned low = ~0u;
      for (int base = 0; base < done; base += 32) low = min(low, lds64(slots + 8 * min(base + lane, done - 1)).y);
      low = __reduce_min_sync(FULL, low);
      t = bound(0, done, m, 32, (unsigned long long)low << 32);
    }
    int n = 0;
    for (int base = 0; base < done; base += 32) {
      const int i = base + lane;
      const unsigned long long k = slot(min(i, done - 1));
      const bool in = i < done && k < t;
      const unsigned b = __ballot_sync(FULL, in);
      const int at = n + __popc(b & lower);
      if (in && at < 32) sts64(scratch + 8 * at, (unsigned)k, (unsigned)(k >> 32));
      n += __popc(b);
    }
    return sorted_scratch(min(n, 32));
  }
  // Slots 0 .. done - 1 in ascending order: a bitonic network whose comparators all point upwards, so that it works for
  // any number of keys.
  __device__ __forceinline__ void sort_done() const {
    __syncwarp();
    for (int size = 2; size < 2 * done; size *= 2) {
      for (int half = size / 2, lg = __ffs(half) - 1; half > 0; half /= 2, --lg) {
        // pairs (i, j): the first stage of a merge pairs a block's keys from both ends, the others half a block apart
        const int pairs = ((done + 2 * half - 1) >> (lg + 1)) << lg;
        for (int base = 0; base < pairs; base += 32) {
          const int p = base + lane;
          const int start = (p >> lg) << (lg + 1), off = p & (half - 1);
          const int i = start + off;
          const int j = 2 * half == size ? start + 2 * half - 1 - off : i + half;
          if (j < done) {
            const unsigned long long a = slot(i), b = slot(j);
            if (b < a) {
              set_slot(i, b);
              set_slot(j, a);
            }
          }
        }
        __syncwarp();
      }
    }
  }
};

// ---------------------------------------------------------------------------
// results of a search
// ---------------------------------------------------------------------------
// Where a search leaves rank j of query qi: slots past the last key read -1 / +inf.
__device__ __forceinline__ void write_result(const SearchParams& p, long long qi, int j, bool have,
                                             unsigned long long k) {
  int id = -1;
  float dist = __int_as_float(0x7f800000);
  if (have) {
    id = key_id(k);
    dist = key_dist(k);
    if (p.labels) id = __ldg(p.labels + id);
  }
  p.out_ids[(size_t)qi * p.topk + j] = id;
  p.out_dist[(size_t)qi * p.topk + j] = dist;
}

// Ascending top-k of what the walk expanded; found = min(their number, k).
__device__ __forceinline__ void write_closest(const SearchParams& p, long long qi, Frontier& fr) {
  const int found = min(fr.done, p.topk);
  if (p.topk <= 32) {
    const unsigned long long k = fr.closest(p.topk);
    if (fr.lane < p.topk) write_result(p, qi, fr.lane, fr.lane < found, k);
  } else {
    fr.sort_done();
    for (int j = fr.lane; j < p.topk; j += 32) write_result(p, qi, j, j < found, fr.slot(min(j, p.slots - 1)));
  }
  if (fr.lane == 0) p.out_found[qi] = found;
  __syncwarp();
}
// The same by all warps of a CTA: each takes 32 of the `done` keys at a time and counts the smaller ones, which is a key's rank, as
// keys are different.  For more than 32 results of few queries, whose other warps are many and idle.
// Against the slots sorted in place by warp 0, 16 warps: two queries of 300 000 x 50 for 100 results, ef 128 and 400, 141.9 / 140.0 and 229.4 / 217.8 us.
// (With four warps it gains nothing, and the code costs rows of 300 floats 3 %.)
__device__ __forceinline__ void write_ranked(const SearchParams& p, long long qi, const Frontier& fr, int done, int w,
                                             int warps) {
  for (int base = 32 * w; base < done; base += 32 * warps) {
    const int i = base + fr.lane;
    const unsigned long long k = fr.slot(min(i, done - 1));
    int rank = 0;
    for (int j = 0; j < done; j += 2) {
      const uint4 v = lds128(fr.slots + 8 * j);  // (the number of slots is even)
      rank += Frontier::word(make_uint2(v.x, v.y)) < k ? 1 : 0;
      rank += j + 1 < done && Frontier::word(make_uint2(v.z, v.w)) < k ? 1 : 0;
    }
    if (i < done && rank < p.topk) write_result(p, qi, rank, true, k);
  }
  for (int j = done + 32 * w + fr.lane; j < p.topk; j += 32 * warps) write_result(p, qi, j, false, 0ull);
  if (w == 0 && fr.lane == 0) p.out_found[qi] = min(done, p.topk);
}

}  // namespace hnsw
