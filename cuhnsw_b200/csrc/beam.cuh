// Warp-level building blocks of the graph walk: a sorted candidate/result list
// in shared memory, a lossy visited table, the ef-bounded best-first search of
// one layer and the greedy descent through the upper layers.
//
// What they replace in the reference:
//   sorted list + batch merge   PqPush/PqPop (cpp/include/cuda_heap_kernels.cuh:13-49, thread 0 only,
//                               heap in global memory), GetCand (cuda_utils_kernels.cuh:104-151) and
//                               CheckAlreadyExists (cuda_utils_kernels.cuh:50-103)
//   visited table               CheckVisited (cuda_utils_kernels.cuh:185-210)
//   beam_layer                  the expansion loops of SearchGraphKernel (cuda_search_kernels.cuh:114-139)
//                               and BuildLevelGraphKernel (cuda_build_kernels.cuh:219-248)
//   greedy_descent              GetEntryPointsKernel (cuda_search_kernels.cuh:22-66)
//
// One warp owns one query; there is no block-level synchronisation anywhere.
#pragma once
#include "common.cuh"
#include "distance.cuh"
#include "kernels.h"
#include "smem.cuh"

namespace hnsw {

__device__ __forceinline__ VecTable make_table(const GraphView& g) {
  return VecTable{static_cast<const unsigned char*>(g.vec), (unsigned)g.vstride * (g.rows16 ? 2u : 4u), (g.d + 3) / 4, g.d,
                  g.dist_type};
}

struct WalkCounters {  // per warp and launch
  unsigned evals;       // rows gathered for a distance
  unsigned expansions;  // adjacency rows read at the searched layer
  unsigned sweeps;      // adjacency rows read during greedy descent
  unsigned inserts;     // keys merged into the list
};

// Number of bits that hold every node id of an index with n nodes.
__host__ __device__ inline int id_bits(long long n) {
  int b = 1;
  while (b < 31 && (1ll << b) < n) ++b;
  return b;
}
// Bits that tell the ids of one bucket apart: those of ceil(2^B / buckets) values, B = id_bits(n).
__host__ __device__ inline int visited_tag_bits(long long n, int buckets) {
  int t = id_bits(n);
  while (t > 0 && buckets > 1) {
    buckets >>= 1;
    --t;
  }
  return t;
}

// Lossy set of node ids in shared memory with no false positives.  id -> h = id * odd mod 2^B is a bijection on B-bit
// numbers.  Bucket b, of any number of buckets, holds the range of h with floor(h * buckets / 2^B) = b, whose low bits, the
// tag, differ, so (bucket, tag) identifies the id exactly and only the tag has to be stored, with one more bit that says that
// there is one.  Each bucket keeps its four most recent tags; a displaced id is evaluated again when it comes
// back, which is never a different result: WarpList turns it down when merging, Frontier looks it up (an id that is not in
// the table can only have been there if its bucket is full), and a key that left the list can never re-enter.
// Four tags per bucket instead of two in the same space, tested two at a time: evaluations per query at 1.18 M x 50, ef 200
// and 400, 1173 -> 1075 and 1545 -> 1288 (1027 distinct rows at ef 200), at 1 M x 128, ef 256, 3887 -> 3624.
struct VisitedTable {
  unsigned vt;       // shared-memory address: buckets of four tags, the newest first (4 x 16 or 4 x 32 bit)
  unsigned mul;      // odd << (32 - B): id * mul is h in the upper B bits
  int shift;         // 32 - B
  unsigned buckets;
  unsigned tag_mask;
  bool wide;         // 32-bit tags
  int vbytes;

  // bytes for `entries` tags, a multiple of 16: 2 per tag where 15 bits tell the ids of a bucket apart, else 4
  __host__ __device__ static bool needs_wide(int entries, long long n) { return visited_tag_bits(n, buckets_of(entries)) > 15; }
  __host__ __device__ static size_t smem_bytes(int entries, long long n) {
    return ((size_t)buckets_of(entries) * (needs_wide(entries, n) ? 16 : 8) + 15) / 16 * 16;
  }
  __host__ __device__ static int buckets_of(int entries) { return entries >= 8 ? entries / 4 : 1; }
  __device__ __forceinline__ void bind_table(unsigned smem, int entries, long long n) {
    const int b = buckets_of(entries);
    vt = smem;
    buckets = (unsigned)b;
    shift = 32 - id_bits(n);
    mul = 2654435761u << shift;
    const int tag_bits = visited_tag_bits(n, b);
    tag_mask = (1u << tag_bits) - 1u;
    wide = tag_bits > 15;
    vbytes = (b * (wide ? 16 : 8) + 15) / 16 * 16;
  }
  // empties the table; warp w of `warps` does its share
  __device__ __forceinline__ void clear(int w, int warps) {
    for (int i = w * 32 + lane_id(); i < vbytes / 16; i += warps * 32) sts128(vt + 16 * i, 0u, 0u, 0u, 0u);
  }
  // not zero exactly if one of the halves of v is zero
  static __device__ __forceinline__ unsigned zero_half(unsigned v) { return (v - 0x00010001u) & ~v & 0x80008000u; }
  // Is the id in the table?  Any value may be asked for; no branch but the one on the table's kind, so that a warp
  // with a few live lanes runs straight through.
  __device__ __forceinline__ bool knows(int id) const {
    const unsigned g = (unsigned)id * mul, b = __umulhi(g, buckets);
    const unsigned tag = (g >> shift) & tag_mask;
    if (!wide) {
      const uint2 w = lds64(vt + 8 * b);
      const unsigned t = (tag | 0x8000u) * 0x10001u;
      return (zero_half(w.x ^ t) | zero_half(w.y ^ t)) != 0u;
    }
    const uint4 w = lds128(vt + 16 * b);
    const unsigned t = tag | 0x80000000u;
    return w.x == t || w.y == t || w.z == t || w.w == t;
  }
  // What the table said of an id: `full`: if it is not known, it may have been forgotten.
  struct Seen {
    unsigned at, tag;
    bool known, full;
  };
  // an id that is not there enters if `on`
  __device__ __forceinline__ Seen enter(int id, bool on) {
    const unsigned g = (unsigned)id * mul, b = __umulhi(g, buckets);
    const unsigned tag = (g >> shift) & tag_mask;
    Seen s;
    if (!wide) {
      s.at = vt + 8 * b;
      s.tag = tag | 0x8000u;
      const uint2 w = lds64(s.at);
      const unsigned t = s.tag * 0x10001u;
      s.known = (zero_half(w.x ^ t) | zero_half(w.y ^ t)) != 0u;
      s.full = w.y >> 31;
      if (on && !s.known) put(s, w);
    } else {
      s.at = vt + 16 * b;
      s.tag = tag | 0x80000000u;
      const uint4 w = lds128(s.at);
      s.known = w.x == s.tag || w.y == s.tag || w.z == s.tag || w.w == s.tag;
      s.full = w.w != 0u;
      if (on && !s.known) sts128(s.at, s.tag, w.x, w.y, w.z);
    }
    return s;
  }
  __device__ __forceinline__ void put(const Seen& s, uint2 w) const {
    sts64(s.at, (w.x << 16) | s.tag, __funnelshift_l(w.x, w.y, 16));
  }
  // Behind a __syncwarp: ids that entered a bucket together with others, of which one was stored, enter again until they
  // are there or their bucket is full.
  __device__ __forceinline__ void settle(const Seen& s, bool entered) {
    const unsigned newest = lds32(s.at);
    if (!__any_sync(FULL, entered && (wide ? newest : newest & 0xffffu) != s.tag)) return;
    for (;;) {
      bool missing;
      if (!wide) {
        const uint2 w = lds64(s.at);
        const unsigned t = s.tag * 0x10001u;
        missing = entered && (zero_half(w.x ^ t) | zero_half(w.y ^ t)) == 0u && !(w.y >> 31);
        if (!__any_sync(FULL, missing)) return;
        if (missing) put(s, w);
      } else {
        const uint4 w = lds128(s.at);
        missing = entered && w.x != s.tag && w.y != s.tag && w.z != s.tag && w.w == 0u;
        if (!__any_sync(FULL, missing)) return;
        if (missing) sts128(s.at, s.tag, w.x, w.y, w.z);
      }
      __syncwarp();
    }
  }
  __device__ __forceinline__ bool test_and_set(int id, bool on = true) { return enter(id, on).known; }
};

// The same with two tags per bucket, a power of two of buckets, and ~0 for no tag: what a walk on a list of keys needs, which
// turns down an id that comes twice by itself.  It forgets more (evaluations per query above), but tests a bucket in one
// word.  Which of the two is a matter of the registers that the rest of a kernel leaves; one B200, ms, two / four tags:
//   one warp per query, fp32 rows of 65 to 96 values (40 000 queries, ef 128, of 620 187 x 72, 400 000 x 80, 400 000 x 96) 2.76 / 2.93,
//   3.65 / 3.80, 2.66 / 2.81, and rows of more than 128 (8000, ef 128, of 200 000 x 150, x 300 and x 500 f16) 1.11 / 1.15, 1.25 / 1.30,
//   1.28 / 1.36: two.  Rows of up to 64 values (40 000 of 1.18 M x 50) 2.55 / 2.49, 97 to 128 (600 000 x 128) 5.12 / 4.91, 96 bfloat16
//   2.58 / 2.51: four.
//   one CTA per query on a list: 1000 of 200 000 x 32, ef 128 and 200 0.318 / 0.360 and 0.415 / 0.460, of 200 000 x 128, ef 128, 0.519 /
//   0.530: two.
struct VisitedPairs {
  unsigned vt;     // shared-memory address: buckets of two tags (2 x 16 bit in one word, or 2 x 32 bit)
  unsigned hmask;  // 2^B - 1, B = id_bits(n)
  int tag_bits;    // low bits of the hash kept as the tag; the rest is the bucket number
  unsigned tag_mask;
  bool wide;       // 32-bit tags
  int vbytes;

  __host__ __device__ static bool needs_wide(int entries, long long n) { return visited_tag_bits(n, entries / 2) > 15; }
  __host__ __device__ static size_t smem_bytes(int entries, long long n) {
    return (size_t)entries * (needs_wide(entries, n) ? 4 : 2);
  }
  __device__ __forceinline__ void bind_table(unsigned smem, int entries, long long n) {
    vt = smem;
    hmask = (1u << id_bits(n)) - 1u;
    tag_bits = visited_tag_bits(n, entries / 2);
    tag_mask = (1u << tag_bits) - 1u;
    wide = tag_bits > 15;
    vbytes = entries * (wide ? 4 : 2);
  }
  // empties the table; warp w of `warps` does its share
  __device__ __forceinline__ void clear(int w, int warps) {
    for (int i = w * 32 + lane_id(); i < vbytes / 16; i += warps * 32) sts128(vt + 16 * i, ~0u, ~0u, ~0u, ~0u);
  }
  // Is the id in the table?  Any value may be asked for; no branch but the one on the table's kind, so that a warp
  // with a few live lanes runs straight through.
  __device__ __forceinline__ bool knows(int id) const {
    const unsigned h = ((unsigned)id * 2654435761u) & hmask;
    const unsigned tag = h & tag_mask;
    if (!wide) {
      const unsigned x = lds32(vt + 4 * (h >> tag_bits)) ^ (tag * 0x10001u);
      return (x & 0xffffu) == 0u || x < 0x10000u;
    }
    const uint2 w = lds64(vt + 8 * (h >> tag_bits));
    return w.x == tag || w.y == tag;
  }
  // the same, and an id that is not there enters if `on`
  __device__ __forceinline__ bool test_and_set(int id, bool on = true) {
    const unsigned h = ((unsigned)id * 2654435761u) & hmask;
    const unsigned tag = h & tag_mask;
    if (!wide) {
      const unsigned at = vt + 4 * (h >> tag_bits);
      const unsigned w = lds32(at), x = w ^ (tag * 0x10001u);
      const bool known = (x & 0xffffu) == 0u || x < 0x10000u;
      if (on && !known) sts32(at, (w << 16) | tag);
      return known;
    }
    const unsigned at = vt + 8 * (h >> tag_bits);
    const uint2 w = lds64(at);
    const bool known = w.x == tag || w.y == tag;
    if (on && !known) sts64(at, tag, w.x);
    return known;
  }
};

// key i of an array of keys in shared memory
__device__ __forceinline__ unsigned long long key_at(unsigned keys, int i) {
  const uint2 w = lds64(keys + 8 * i);
  return ((unsigned long long)w.y << 32) | w.x;
}

// Per-warp shared-memory state.  Loop bounds and branch conditions come from ballots, shuffles and reductions rather than
// from loads, so that the compiler knows them to be the same in every lane (figures in smem.cuh).
template <class Table>
struct WarpList : Table {
  unsigned keys;  // shared-memory address of `cap` 64-bit keys, ascending (distance, id)
  unsigned spos;  // 32 words of scratch
  int cap;
  int size;
  int cursor;  // every key before `cursor` is expanded
  unsigned long long worst;  // largest key of a full list, KEY_MAX while there is room

  __host__ __device__ static size_t smem_bytes(int cap, int entries, long long n) {
    return (size_t)((cap + 31) / 32 * 32) * 8 + 32 * 4 + Table::smem_bytes(entries, n);
  }
  __device__ __forceinline__ void bind(void* smem, int cap_, int entries, long long n) {
    keys = kept(smem_addr(smem));
    const int capr = (cap_ + 31) / 32 * 32;
    spos = keys + 8 * capr;
    this->bind_table(spos + 32 * 4, entries, n);
    cap = cap_;
    size = 0;
    cursor = 0;
    worst = KEY_MAX;
  }
  // key i with its flag
  __device__ __forceinline__ unsigned long long key(int i) const { return key_at(keys, i); }
  __device__ __forceinline__ void set_key(int i, unsigned long long k) const {
    sts64(keys + 8 * i, (unsigned)k, (unsigned)(k >> 32));
  }
  // low words (id and flag) of two neighbouring keys, the same in every lane
  __device__ __forceinline__ uint2 low_words(int i) const {
    const unsigned w = lds32(keys + 8 * (i + (lane_id() & 1)));
    return make_uint2(__shfl_sync(FULL, w, 0), __shfl_sync(FULL, w, 1));
  }
  __device__ __forceinline__ void flag_key(int i, unsigned low) const {
    if (lane_id() == 0) sts32(keys + 8 * i, low | (unsigned)KEY_FLAG);
    __syncwarp();
  }
  // The table size is proportional to the list capacity, so clearing it is
  // O(nodes touched); the reference resets through a touched-slot list
  // (cuda_search_kernels.cuh:145-147).
  __device__ __forceinline__ void reset() {
    this->clear(0, 1);
    size = 0;
    cursor = 0;
    worst = KEY_MAX;
    __syncwarp();
  }
  __device__ __forceinline__ void mark(int id) {
    if (lane_id() == 0) this->test_and_set(id);
    __syncwarp();
  }

  // Merges up to 32 new keys (one per lane, `active` lanes) into the list,
  // keeping the `cap` smallest.  Equivalent to inserting them one by one in any
  // order with "insert if not full or smaller than the largest, evicting the
  // largest" (cuda_utils_kernels.cuh:220-225).  Returns the smallest position a
  // newcomer took, or `cap` when nothing was inserted.
  __device__ __forceinline__ int merge(unsigned long long nk, bool active, WalkCounters& wc) {
    const int lane = lane_id();
    bool keep = active && nk < worst;
    const unsigned km0 = __ballot_sync(FULL, keep);
    if (km0 == 0) return cap;
    // pos = number of list keys smaller than the new key
    int pos = 0;
    bool dup = false;
    const int nch = (size + 31) >> 5;
    if (__popc(km0) <= 4 && nch <= 32) {
      // up to four newcomers: two-level search by the whole warp, one newcomer at a time
      const unsigned long long pv = (lane < nch) ? (key(min(lane * 32 + 31, size - 1)) & KEY_MASK) : KEY_MAX;
      for (unsigned mm = km0; mm; mm &= mm - 1) {
        const int b = __ffs(mm) - 1;
        const unsigned long long kb = shfl64(nk, b);
        // chunks entirely below kb (lanes >= nch hold KEY_MAX)
        const int c = nch > 1 ? __popc(__ballot_sync(FULL, pv < kb)) : 0;
        const int i = c * 32 + lane;
        const unsigned long long kv = (i < size) ? (key(i) & KEY_MASK) : KEY_MAX;
        const unsigned lt = __ballot_sync(FULL, kv < kb);
        const unsigned eq = __ballot_sync(FULL, kv == kb);
        if (lane == b) {
          pos = min(c * 32 + __popc(lt), size);
          dup = eq != 0;
        }
      }
    } else if (__popc(km0) <= 4) {
      // the same for lists of more than 1024 keys: a lane stands for a span of `cs` chunks, the span that holds
      // the newcomer's place is then searched chunk by chunk
      const int cs = (nch + 31) >> 5;
      for (unsigned mm = km0; mm; mm &= mm - 1) {
        const int b = __ffs(mm) - 1;
        const unsigned long long kb = shfl64(nk, b);
        const unsigned long long pv = (lane * cs < nch) ? (key(min((lane + 1) * cs * 32 - 1, size - 1)) & KEY_MASK) : KEY_MAX;
        const int c = __popc(__ballot_sync(FULL, pv < kb));  // spans entirely below kb
        int below = 0;
        bool same = false;
        for (int j = 0; j < cs; ++j) {
          const int i = (c * cs + j) * 32 + lane;
          const unsigned long long kv = (i < size) ? (key(i) & KEY_MASK) : KEY_MAX;
          const unsigned lt = __ballot_sync(FULL, kv < kb);
          same = same || __ballot_sync(FULL, kv == kb) != 0;
          below += __popc(lt);
          if (lt != 0xffffffffu) break;  // the place is in this chunk
        }
        if (lane == b) {
          pos = min(c * cs * 32 + below, size);
          dup = same;
        }
      }
    } else {
      int lo = 0, hi = keep ? size : 0;
      while (__any_sync(FULL, lo < hi)) {
        if (lo < hi) {
          int mid = (lo + hi) >> 1;
          if ((key(mid) & KEY_MASK) < nk) lo = mid + 1;
          else hi = mid;
        }
      }
      pos = lo;
      dup = keep && pos < size && (key(pos) & KEY_MASK) == nk;
    }
    if (dup) keep = false;  // already listed
    const unsigned km = __ballot_sync(FULL, keep);
    if (km == 0) return cap;
    const int m = __popc(km);
    int minpos;
    if (m == 1) {
      // the common case: one newcomer, everything from its position on moves up by one
      minpos = __shfl_sync(FULL, pos, __ffs(km) - 1);
      // windows of 64 keys, top down; both halves are read before either is written (a window's
      // targets lie above everything a lower window reads)
      for (int hi = size; hi > minpos; hi -= 64) {
        const int i = hi - 32 + lane, i2 = i - 32;
        const bool have = i >= minpos, have2 = i2 >= minpos;
        const unsigned at = keys + 8 * i;
        const uint2 v = lds64(have ? at : keys);
        const uint2 v2 = lds64(have2 ? at - 256 : keys);
        __syncwarp();
        if (have && i + 1 < cap) sts64(at + 8, v.x, v.y);
        if (have2) sts64(at - 248, v2.x, v2.y);  // i2 + 1 <= size - 32 < cap
      }
      if (keep) set_key(pos, nk);  // pos < cap: either the list is not full or nk < worst
    } else {
      int rk = 0;
      for (unsigned mm = km; mm; mm &= mm - 1) {
        const int b = __ffs(mm) - 1;
        const unsigned long long kb = shfl64(nk, b);
        rk += (kb < nk) ? 1 : 0;
      }
      if (keep) sts32(spos + 4 * rk, (unsigned)pos);  // newcomer positions, ascending
      minpos = (int)__reduce_min_sync(FULL, keep ? (unsigned)pos : 0x7fffffffu);
      __syncwarp();
      const int mypos = (lane < m) ? (int)lds32(spos + 4 * lane) : 0x7fffffff;
      for (int hi = size; hi > minpos; hi -= 64) {
        // key i moves up by the number of newcomers placed at or before it; that number is the same for a
        // whole window of 32 unless a newcomer lands inside it.  Two windows per turn, both read before
        // either is written.
        const int i = hi - 32 + lane, i2 = i - 32;
        const bool have = i >= minpos, have2 = i2 >= minpos;
        const unsigned at = keys + 8 * i;
        const uint2 v = lds64(have ? at : keys);
        const uint2 v2 = lds64(have2 ? at - 256 : keys);
        const int below2 = __popc(__ballot_sync(FULL, mypos <= hi - 64));
        const int below = __popc(__ballot_sync(FULL, mypos <= hi - 32));
        const int upto = __popc(__ballot_sync(FULL, mypos <= hi - 1));
        int cnt = below, cnt2 = below2;
        for (int j = below; j < upto; ++j) cnt += ((int)lds32(spos + 4 * j) <= i) ? 1 : 0;
        for (int j = below2; j < below; ++j) cnt2 += ((int)lds32(spos + 4 * j) <= i2) ? 1 : 0;
        __syncwarp();
        if (have && i + cnt < cap) sts64(at + 8 * cnt, v.x, v.y);
        if (have2 && i2 + cnt2 < cap) sts64(at - 256 + 8 * cnt2, v2.x, v2.y);
      }
      if (keep && pos + rk < cap) set_key(pos + rk, nk);
    }
    size = min(cap, size + m);
    cursor = min(cursor, minpos);
    wc.inserts += m;
    __syncwarp();
    worst = (size >= cap) ? (key(cap - 1) & KEY_MASK) : KEY_MAX;
    return minpos;
  }

  // list = {k}
  __device__ __forceinline__ void seed(unsigned long long k) {
    if (lane_id() == 0) set_key(0, k);
    size = 1;
    cursor = 0;
    worst = cap <= 1 ? (k & KEY_MASK) : KEY_MAX;
    __syncwarp();
  }

  // moves `cursor` to the first unexpanded key at or after it
  __device__ __forceinline__ void advance() {
    const int lane = lane_id();
    int c = cursor;
    while (c < size) {
      int i = c + lane;
      bool open = (i < size) && !(lds32(keys + 8 * i) & (unsigned)KEY_FLAG);
      unsigned m = __ballot_sync(FULL, open);
      if (m) {
        c += __ffs(m) - 1;
        break;
      }
      c += 32;
    }
    cursor = min(c, size);
  }
};

// One chunk of an adjacency row (lane l holds the id in slot l, -1 = unused): filter through the
// visited table, evaluate the fresh ids, merge them.
template <class Dist, class List>
__device__ __forceinline__ int expand_chunk(Dist& de, List& wl, int nid, int self, WalkCounters& wc) {
  const int lane = lane_id();
  bool fresh = (nid >= 0) && (nid != self);
  fresh = !wl.test_and_set(nid, fresh) && fresh;
  const unsigned fm = __ballot_sync(FULL, fresh);
  if (fm == 0) return wl.cap;
  const int n = __popc(fm);
  if (fresh) sts32(wl.spos + 4 * __popc(fm & ((1u << lane) - 1)), (unsigned)nid);
  __syncwarp();
  const int cid = (int)lds32(wl.spos + 4 * lane);
  // the shuffles inside eval() order this read before any later write of spos
  const float dist = de.eval(cid, n);
  wc.evals += n;
  return wl.merge(mkkey(dist, cid), lane < n, wc);
}

// Whole adjacency row; `rows` is a sentinel-padded table: unused slots hold -1.
template <class Dist, class List>
__device__ __forceinline__ void expand_row(Dist& de, List& wl, const int* __restrict__ row, int stride,
                                           int self, WalkCounters& wc) {
  const int lane = lane_id();
  for (int base = 0; base < stride; base += 32) {
    const int l = base + lane;
    const int nid = (l < stride) ? __ldg(row + l) : -1;
    expand_chunk(de, wl, nid, self, wc);
  }
}

// Row number of node `id` in the adjacency table of `level`: layer 0 is indexed by id,
// the upper layers of a node are stored consecutively from upper_base[id].
__device__ __forceinline__ size_t row_index(const int* __restrict__ upper_base, int level, int id) {
  return level == 0 ? (size_t)id : (size_t)__ldg(upper_base + id) + (size_t)(level - 1);
}

// The same as 32 bits, and the row of that number: one multiplication and addition per address instead of products of
// 64 bits (with those of the vectors' addresses: 10 000 queries x 50, ef 200, 1.42 -> 1.31 ms).
__device__ __forceinline__ unsigned row_number(const int* __restrict__ upper_base, int level, int id) {
  return level == 0 ? (unsigned)id : (unsigned)(__ldg(upper_base + id) + (level - 1));
}
__device__ __forceinline__ const int* row_at(const int* __restrict__ rows, unsigned number, int stride) {
  return reinterpret_cast<const int*>(reinterpret_cast<const char*>(rows) + (size_t)number * (4u * (unsigned)stride));
}

// ef-bounded best-first search of one layer.  The list must already hold the
// seeds; on return it holds the min(ef, reachable) closest nodes, ascending.
// While the neighbours of the current node are gathered, the first 32 slots of
// the adjacency row of the likely next node (the key after the cursor) are
// already on their way; a newcomer that overtakes it costs one ordinary load.
template <class Dist, class List>
__device__ __forceinline__ void beam_layer(Dist& de, List& wl, const int* __restrict__ rows, int stride,
                                           const int* __restrict__ upper_base, int level, int self,
                                           WalkCounters& wc) {
  const int lane = lane_id();
  int pf_node = -1, pf_val = -1;
  wl.advance();
  if (wl.cursor >= wl.size) return;
  // low words of the closest unexpanded key and of the key after it
  uint2 k = wl.low_words(wl.cursor);
  for (;;) {
    const int at = wl.cursor;  // position of the key being expanded; insertions at or before it move the cursor
    const unsigned k2 = at + 1 < wl.size ? k.y : (unsigned)KEY_FLAG;
    wl.flag_key(at, k.x);
    const int cur = (int)(k.x & 0x7fffffffu);
    const int* row = row_at(rows, row_number(upper_base, level, cur), stride);
    int nid;
    if (cur == pf_node) {
      nid = pf_val;
    } else {
      nid = (lane < stride) ? __ldg(row + lane) : -1;
    }
    pf_node = -1;
    const bool open2 = !(k2 & (unsigned)KEY_FLAG);
    if (open2) {
      pf_node = (int)k2;
      const int* nrow = row_at(rows, row_number(upper_base, level, pf_node), stride);
      pf_val = (lane < stride) ? __ldg(nrow + lane) : -1;
    }
    wc.expansions += 1;
    int first_new = expand_chunk(de, wl, nid, self, wc);
    for (int base = 32; base < stride; base += 32) {
      const int l = base + lane;
      first_new = min(first_new, expand_chunk(de, wl, (l < stride) ? __ldg(row + l) : -1, self, wc));
    }
    // next key: a newcomer placed at or before at + 1, else the old successor if it is still unexpanded,
    // else scan on
    if (first_new > at + 1 && open2) {
      // no newcomer in front of the old successor: it sits at at + 1 unchanged
      wl.cursor = at + 1;
    } else {
      __syncwarp();
      wl.advance();
      if (wl.cursor >= wl.size) break;
    }
    k = wl.low_words(wl.cursor);
  }
}

// The adjacency rows of one layer, for a warp whose lanes read a slot each.
struct LayerRows {
  const int* mine;  // this lane's slot of row 0
  int stride;       // slots
  const int* upper_base;
  int level;
  int lane;

  __device__ __forceinline__ LayerRows() {}
  __device__ __forceinline__ LayerRows(const int* rows, int stride_, const int* upper_base_, int level_) {
    lane = lane_number();
    mine = rows + lane;
    stride = stride_;
    upper_base = upper_base_;
    level = level_;
  }
  __device__ __forceinline__ const int* row(int id) const {
    return row_at(mine, row_number(upper_base, level, id), stride);
  }
  // slot base + lane of the row at p
  __device__ __forceinline__ int read(const int* p, int base) const {
    return base + lane < stride ? __ldg(p + base) : -1;
  }
};

// reverse_cand variant (cuda_utils_kernels.cuh:113-124 of the reference): every step expands
// the FARTHEST unexpanded key of the list; the walk ends when every key is expanded.
template <class Dist, class List>
__device__ __forceinline__ void beam_layer_reverse(Dist& de, List& wl, const int* __restrict__ rows, int stride,
                                                   const int* __restrict__ upper_base, int level, int self,
                                                   WalkCounters& wc) {
  const int lane = lane_id();
  int hi = wl.size - 1;  // every key above `hi` is expanded
  for (;;) {
    int at = -1;
    for (int base = hi & ~31; hi >= 0 && base >= 0; base -= 32) {
      const int i = base + lane;
      const bool open = (i <= hi) && !(lds32(wl.keys + 8 * i) & (unsigned)KEY_FLAG);
      const unsigned m = __ballot_sync(FULL, open);
      if (m) {
        at = base + 31 - __clz(m);
        break;
      }
    }
    if (at < 0) break;
    const unsigned k = wl.low_words(at).x;
    __syncwarp();
    wl.flag_key(at, k);
    const int* row = rows + row_index(upper_base, level, (int)k) * stride;
    wc.expansions += 1;
    int first_new = wl.cap;
    for (int base = 0; base < stride; base += 32) {
      const int l = base + lane;
      first_new = min(first_new, expand_chunk(de, wl, (l < stride) ? __ldg(row + l) : -1, self, wc));
    }
    __syncwarp();
    hi = (first_new < wl.cap) ? wl.size - 1 : at - 1;
  }
}

// Greedy walk through layers top..bottom+1: in each layer, evaluate every
// neighbour of the current node, move to the closest one if it is strictly
// closer (first in row order among equals), repeat until no move.  Rows are
// packed.  Where a neighbour's own rows begin is read beside its vector, so that a
// move does not wait for it.
template <class Dist>
__device__ __forceinline__ void greedy_descent(Dist& de, const int* __restrict__ rowsU, int strideU,
                                               const int* __restrict__ upper_base, int top, int bottom_excl,
                                               int& cur, float& dcur, WalkCounters& wc) {
  const int lane = lane_id();
  if (top <= bottom_excl) return;
  int first = __ldg(upper_base + cur);  // the node's row on layer 1
  for (int l = top; l > bottom_excl; --l) {
    bool moved = true;
    while (moved) {
      moved = false;
      const int* row = rowsU + ((size_t)first + (l - 1)) * strideU;
      float best_d = dcur;
      wc.sweeps += 1;
      for (int base = 0; base < strideU; base += 32) {
        const int li = base + lane;
        const int nid = (li < strideU) ? __ldg(row + li) : -1;
        const unsigned fm = __ballot_sync(FULL, nid >= 0);
        if (fm == 0) break;
        const int n = __popc(fm);
        const int begin = nid >= 0 ? __ldg(upper_base + nid) : 0;
        const float dist = de.eval(nid, n);
        wc.evals += n;
        // closest, the first in row order among equals; a NaN is never closest
        const unsigned image = lane < n && dist == dist ? f2ord(dist) : ~0u;
        const unsigned least = __reduce_min_sync(FULL, image);
        const int at = __ffs(__ballot_sync(FULL, image == least)) - 1;
        const int id = __shfl_sync(FULL, nid, at), next = __shfl_sync(FULL, begin, at);
        if (least != ~0u && ord2f(least) < best_d) {
          best_d = ord2f(least);
          cur = id;
          first = next;
          moved = true;
        }
      }
      dcur = best_d;
    }
  }
}

}  // namespace hnsw
