// Binary radix trees built a tile at a time, bottom up, with their boxes.
//
// The tree over sorted keys follows from the prefix lengths d(s) = lcp(key s, key s + 1) of
// neighbouring keys alone: the node whose children meet at split s covers the leaves between
// the nearest splits on either side with a smaller d, and it is the left child of the right one
// of these two if that has the larger d, else the right child of the left one (Karras 2012,
// Apetrei 2014).  No two splits of one node's range share its smallest d, since keys are unique
// once equal ones are told apart by their index.
//
// A block takes kTile consecutive leaves.  Every split inside finds its two neighbours by a
// descent through a table of range minima in shared memory; a node is closed when both lie
// within the tile, borders included, and then its whole subtree does too.  What is left of a
// tile are its largest closed subtrees, in order: they hang off the paths to its two borders, so
// they are few: the splits along a border's path have ever smaller prefixes, 97 lengths at most, so
// there are no more than 2 x 97 + 1 subtrees (for 256 leaves usually about a dozen).  The block that
// finishes last of kFan neighbouring ones takes their lists as its next tiles, subtrees in the
// place of leaves, and so on up to the root, all within one launch.  Only that block reads what
// the others wrote, behind one fence and counter per group, where a climb with an arrival counter
// per node pays a fence and three dependent round trips for every node of the longest path.
//
// Karras' numbering (BVHSource/BVHSoAKernels.cu:7-99): leaf i is node i; an internal node has
// number n + the end of its range next to its sibling -- its last leaf when it is a left child,
// its first when it is a right child or the root.
#pragma once
#include <cuda/atomic>

#include "ar_internal.cuh"
#include "ar_lbvh.cuh"

namespace ar_tree {

constexpr int kTile = 256;  // leaves or subtrees per tile, one thread each
constexpr int kLevels = 8;  // range minima over up to 2^7 splits
constexpr int kFan = 16;    // lists per group

// Scratch between the blocks: the lists, from each tile's first leaf's place on, the boxes of the
// listed nodes by number, a length and an arrival count per list (zero between launches).
struct Scratch {
  int2* open;       // first and last leaf of a listed subtree; n entries
  float4* pending;  // two per node; 2 n entries
  int* length;      // lists_for(n)
  int* arrived;     // lists_for(n)
};
// Lists of all levels for n leaves.
inline long lists_for(long n) {
  long units = (n + kTile - 1) / kTile, total = units + 1;
  while (units > 1) {
    units = (units + kFan - 1) / kFan;
    total += units;
  }
  return total;
}

struct Box2 {  // a child record of a wide node: (lo.xyz, hi.x), (hi.yz, id, tag)
  float4 a, b;
};

// A tile in shared memory: its subtrees, then the closed nodes by their local number (the
// subtree at the end of their range next to their sibling).
struct Links {
  signed char d[kLevels][kTile + 4];  // d[0][i]: the prefix length before subtree i;
                                      // d[k][i]: the smallest of d[0][i .. i + 2^k - 1]
  int first[kTile], last[kTile];      // leaves of the subtrees
  int id[2 * kTile];
  short parent[2 * kTile];            // the closed parent's local number, else -1
  short child[2][kTile];              // of the closed node of each number: places in this struct
  short lo[kTile], hi[kTile];         // of the closed node of each number: its subtrees, hi past
  int made[kTile];                    // children that arrived at it, plus 1 (0: no such node)
  short top[kTile];                   // place of the largest closed subtree that starts here, -1
  int warp_sum[kTile / 32];
  int prefix[kFan + 1];               // of the group's list lengths
  bool last_of_group;
};
struct Boxes {
  float4 a[2 * kTile], b[2 * kTile];
};

// The node at split t (0 < t < m): the nearest splits with a smaller prefix length.  Returns
// whether both lie in the tile.
__device__ __forceinline__ bool node_at(const Links& s, int t, int m, int* lo, int* hi) {
  const signed char v = s.d[0][t];
  int a = t, b = t + 1;  // the splits a .. b - 1 are known to be at least v
#pragma unroll
  for (int k = kLevels - 1; k >= 0; --k) {
    const int h = 1 << k;
    if (a >= h && s.d[k][a - h] >= v) a -= h;
    if (b + h <= m + 1 && s.d[k][b] >= v) b += h;
  }
  *lo = a - 1;
  *hi = b;
  return a > 0 && b <= m;
}

// The boxes of the closed nodes above subtree c: the second child to arrive at a node merges both
// and climbs on.
__device__ __forceinline__ void climb(Links& s, Boxes& box, int c) {
  float4 a = box.a[c], b = box.b[c];
  int p = s.parent[c];
  for (int guard = 0; guard < kTile && p >= 0; ++guard, p = s.parent[c]) {  // at most kTile - 1 deep
    __threadfence_block();  // this child's record before its arrival
    if (atomicAdd(&s.made[p], 1) == 1) return;
    __threadfence_block();  // its sibling's record after that one's arrival
    const int lc = s.child[0][p], rc = s.child[1][p];
    const bool is_left = lc == c;
    const int o = is_left ? rc : lc;
    const float4 oa = box.a[o], ob = box.b[o];
    const ar_lbvh::Box6 mine{a.x, a.y, a.z, a.w, b.x, b.y}, other{oa.x, oa.y, oa.z, oa.w, ob.x, ob.y};
    const ar_lbvh::Box6 u =
        is_left ? ar_lbvh::merge_boxes(mine, other) : ar_lbvh::merge_boxes(other, mine);
    c = kTile + p;
    a = make_float4(u.lx, u.ly, u.lz, u.hx);
    b = make_float4(u.hy, u.hz, __int_as_float(s.id[c]),
                    __float_as_int(b.w) == __float_as_int(ob.w) ? b.w : __int_as_float(-1));
    box.a[c] = a;
    box.b[c] = b;
  }
}

// Finishes the closed nodes of a tile of m subtrees (first, last, d[0] up to d[0][m] and the
// subtrees' records filled in, a barrier since) and leaves the largest closed subtrees in `top`.
// Every thread of the block calls it.
template <class Sink>
__device__ __forceinline__ void close_nodes(Links& s, Boxes& box, int m, int n, const Sink& out) {
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 1; k < kLevels; ++k) {
    const int h = 1 << (k - 1);
    if (t + 2 * h <= m + 1) {
      const signed char a = s.d[k - 1][t], b = s.d[k - 1][t + h];
      s.d[k][t] = a < b ? a : b;
    }
    __syncthreads();
  }
  int lo = 0, hi = 0, num = 0, lc = 0, rc = 0;
  const bool closed = t > 0 && t < m && node_at(s, t, m, &lo, &hi);
  if (closed) {
    const int dl = s.d[0][lo], dr = s.d[0][hi];
    const bool is_left = dr > dl;
    num = is_left ? hi - 1 : lo;
    const int id = n + (is_left ? s.last[num] : s.first[num]);
    lc = lo == t - 1 ? t - 1 : kTile + t - 1;
    rc = hi - 1 == t ? t : kTile + t;
    s.id[kTile + num] = id;
    s.child[0][num] = (short)lc;
    s.child[1][num] = (short)rc;
    s.lo[num] = (short)lo;
    s.hi[num] = (short)hi;
    s.parent[lc] = s.parent[rc] = (short)num;
    s.made[num] = 1;
    out.made(id, s.d[0][t], dl, dr, s.first[lo]);
  }
  __syncthreads();
  if (t < m) climb(s, box, t);
  __syncthreads();
  // links, by local number, and wide nodes by four threads each
  if (t < m && s.parent[t] >= 0) out.parent_of(s.id[t], s.id[kTile + s.parent[t]]);
  if (s.made[t]) {
    const int id = s.id[kTile + t];
    out.links(id, s.id[s.child[0][t]], s.id[s.child[1][t]]);
    if (s.parent[kTile + t] >= 0) out.parent_of(id, s.id[kTile + s.parent[kTile + t]]);
    else s.top[s.lo[t]] = (short)(kTile + t);
  }
  if (t < m && s.parent[t] < 0) s.top[t] = (short)t;
  for (int i = t; i < 4 * kTile; i += kTile) {
    const int node = i >> 2;
    if (!s.made[node]) continue;
    const int c = s.child[(i >> 1) & 1][node];
    out.wide(s.id[kTile + node] - n, i & 3, i & 1 ? box.b[c] : box.a[c]);
  }
  __syncthreads();
}

// Appends the tile's largest closed subtrees, in order, to the list at `to`, which holds `have`
// already; returns its new length.
__device__ __forceinline__ int list_open(Links& s, const Boxes& box, int m, int n, int2* to,
                                         int have, const Scratch& w) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int c = t < m ? s.top[t] : -1;
  const uint32_t some = __ballot_sync(0xffffffffu, c >= 0);
  if (lane == 0) s.warp_sum[warp] = __popc(some);
  __syncthreads();
  int at = have, total = have;
  for (int i = 0; i < kTile / 32; ++i) {
    if (i < warp) at += s.warp_sum[i];
    total += s.warp_sum[i];
  }
  if (c >= 0) {
    const int last = c < kTile ? s.last[t] : s.last[s.hi[c - kTile] - 1];
    __stcg(to + at + __popc(some & ((1u << lane) - 1)), make_int2(s.first[t], last));
    if (c >= kTile) {
      float4* p = w.pending + 2 * (size_t)(s.id[c] - n);
      __stcg(p, box.a[c]);
      __stcg(p + 1, box.b[c]);
    }
  }
  __syncthreads();
  return total;
}

__device__ __forceinline__ void reset_links(Links& s) {
  const int t = threadIdx.x;
  s.parent[t] = s.parent[kTile + t] = -1;
  s.made[t] = 0;
  s.top[t] = -1;
}

// The tree above a block's tile.  The tile's subtrees are in s (and box), filled in by the caller
// up to d[0]; `sink.leaf(i)` is the record of leaf i, readable once its block has arrived.
template <class Lcp, class Sink>
__device__ __forceinline__ void build_up(Links& s, Boxes& box, int m, int n, const Lcp& lcp,
                                         const Sink& sink, const Scratch& w) {
  const int t = threadIdx.x;
  close_nodes(s, box, m, n, sink);
  int unit = blockIdx.x, units = gridDim.x, lists = 0;  // `lists`: of the levels below
  long span = kTile;                                    // leaves per list
  int length = list_open(s, box, m, n, w.open + (size_t)unit * span, 0, w);
  while (units > 1) {
    const int group = unit / kFan, count = min(kFan, units - group * kFan);
    // the block's boxes, lists and leaves are ordered before its arrival by the barrier and the
    // arrival's release (list_open ends with a barrier), and the others' before the block's reads
    // by the arrival's acquire and the next barrier
    if (t == 0) {
      __stcg(w.length + lists + unit, length);
      __threadfence();
      cuda::atomic_ref<int, cuda::thread_scope_device> a(w.arrived[lists + units + group]);
      s.last_of_group = a.fetch_add(1, cuda::memory_order_acq_rel) == count - 1;
      if (s.last_of_group) w.arrived[lists + units + group] = 0;  // for the next launch
      __threadfence();
    }
    __syncthreads();
    if (!s.last_of_group) return;
    if (t < 32) {  // where each of the group's lists starts in their concatenation
      const int len = t < count ? __ldcg(w.length + lists + group * kFan + t) : 0;
      int x = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (t >= o) x += y;
      }
      if (t < kFan) s.prefix[t + 1] = x;
      if (t == 0) s.prefix[0] = 0;
    }
    __syncthreads();
    const long at = (long)group * kFan * span;  // the group's first leaf, and its list's place
    int have = s.prefix[kFan];
    bool joined = false;  // the lists have become one
    // once through the group's subtrees, a tile at a time; at the top until one is left (a tile
    // leaves at most 195 of 256, so a few passes; the bound only guards against unsorted keys)
    int pass = 0;
    do {
      int kept = 0;
      for (int base = 0; base < have; base += kTile) {
        const int c = min(kTile, have - base);
        reset_links(s);
        if (t < c) {
          const int i = base + t;
          long place = at + i;
          if (!joined) {
            int u = 0;
#pragma unroll
            for (int o = kFan / 2; o > 0; o >>= 1)
              if (s.prefix[u + o] <= i) u += o;
            place = at + u * span + (i - s.prefix[u]);
          }
          const int2 e = __ldcg(w.open + place);
          s.first[t] = e.x;
          s.last[t] = e.y;
          const int dl = lcp(e.x, e.x - 1), dr = lcp(e.y, e.y + 1);
          s.d[0][t] = (signed char)dl;
          if (t == c - 1) s.d[0][c] = (signed char)dr;
          const int number = dr > dl ? e.y : e.x;
          s.id[t] = e.x == e.y ? e.x : n + number;
          Box2 r;
          if (e.x == e.y) {
            r = sink.leaf(e.x);
          } else {
            const float4* p = w.pending + 2 * (size_t)number;
            r = Box2{__ldcg(p), __ldcg(p + 1)};
          }
          box.a[t] = r.a;
          box.b[t] = r.b;
        }
        __syncthreads();  // the tile is read before its place in the list is written over
        close_nodes(s, box, c, n, sink);
        kept = list_open(s, box, c, n, w.open + at, kept, w);
      }
      have = kept;
      joined = true;
    } while (units <= kFan && have > 1 && ++pass < 64);
    lists += units;
    unit = group;
    units = (units + kFan - 1) / kFan;
    span *= kFan;
    length = have;
  }
}

}  // namespace ar_tree
