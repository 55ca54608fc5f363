// (a9) Karras LBVH hierarchy, (a10) leaves, (a11) bottom-up refit, (a12) traversal.
//
// Node numbering is the reference's SoA layout (BVHSource/BVHSoAKernels.cu): leaf i at index
// i, internal node i at n + i, root at n.  Boxes are the reference's 32-byte AABB
// {min.xyz, max.xyz, pad, pad}, read as two float4.
//
// Traversal keeps a short stack and finds what it drops again through the tree's parent links, so
// that no depth is too great (the reference has an int[64] stack).  The visit order is the
// reference's (RB_BVHKernels.cu:145-214): at an internal node, its overlapping leaf children are
// handled left then right, then the walk descends into the left internal child if it overlaps,
// and on the way back up into the right one.  Handling contacts in the same order keeps the float
// sums identical to the reference's.
#include <algorithm>

#include "ar_internal.cuh"
#include "ar_dem.cuh"
#include "ar_lbvh.cuh"

using ar_lbvh::Box;
using ar_lbvh::load_box;
using ar_lbvh::overlap;

namespace {

// ---- Karras 2012 internal nodes (kernelConstructRadixTreeSoA, BVHSoAKernels.cu:7-99) -------
// Over sorted codes the common prefix of two leaves is the smallest of those of the neighbours
// between them.  A tile of kBuildTile nodes puts the prefixes of its neighbours into shared memory
// with their minima over 2^k of them, a byte each, and both of a node's searches (the end of its
// range, then its split) descend through the levels: kBuildLevels steps in shared memory for every
// lane, against as many steps, to global memory, as the warp's longest range takes in the search
// over the codes.  The nodes whose range leaves the tile (at most one per bit of the codes and
// side), and those that unsorted codes give equal neighbours, are gathered and search the codes
// with eight lanes each.  Bound by issued instructions (2^24 points, 30 / 63-bit codes: 399 / 478
// -> 242 / 255 us, 1,000,003: 36 / 42 -> 26 / 28 us; one lane for each gathered node 318 / 339 us,
// tiles of 512 277 / 294 us, the second search from its range's own level 262 / 275 us).
constexpr int kBuildTile = 1024;
constexpr int kBuildThreads = 256;
constexpr int kBuildLevels = 11;  // 2^0 to 2^10 neighbours
// Entry q is the prefix of leaves q - 2 and q - 1 of the tile, plus one, so that 0, where there
// are no leaves, ends every search; entries 0 and kBuildEnd, outside the tile, are 0 too.
constexpr int kBuildEnd = kBuildTile + 2;
constexpr int kBuildRow = kBuildEnd / 4 + 1;  // in words of four entries
static_assert(kBuildTile + 1 < 1 << kBuildLevels, "the descent needs each level once");
template <class Lcp>
__global__ void __launch_bounds__(kBuildThreads) build_kernel(Lcp lcp, int n, ar_lbvh::TreeOut out) {
  __shared__ uint32_t s_words[kBuildLevels][kBuildRow];
  __shared__ uint16_t s_list[kBuildTile];
  __shared__ int s_count;
  const int t0 = blockIdx.x * kBuildTile;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    out.parent[n] = -1;  // root: no parent (the reference leaves it unset)
  if (threadIdx.x == 0) s_count = 0;
  uint8_t* base = reinterpret_cast<uint8_t*>(s_words[0]);
  for (int q = threadIdx.x; q < 4 * kBuildRow; q += kBuildThreads) {
    const int k = t0 - 2 + q;
    base[q] = (uint8_t)(q == 0 || q >= kBuildEnd || k < 0 ? 0 : lcp(k, k + 1) + 1);
  }
  __syncthreads();
#pragma unroll
  for (int lv = 1; lv < kBuildLevels; ++lv) {
    const int half = 1 << (lv - 1);
    for (int w = threadIdx.x; w < kBuildRow; w += kBuildThreads) {
      const uint32_t a = s_words[lv - 1][w];
      const int o = w + (half < 4 ? 1 : half / 4);
      uint32_t b = o < kBuildRow ? s_words[lv - 1][o] : 0u;
      if (half < 4) b = __funnelshift_r(a, b, 8 * half);
      s_words[lv][w] = __vminu4(a, b);
    }
    __syncthreads();
  }
  auto least = [&](int lv, int q) -> int {  // over the entries q .. q + 2^lv - 1
    return base[lv * 4 * kBuildRow + q];
  };
  for (int u = 0; u < kBuildTile / kBuildThreads; ++u) {
    const int q = u * kBuildThreads + threadIdx.x, i = t0 + q;
    if (i >= n - 1) break;
    const int before = least(0, q + 1), after = least(0, q + 2);
    const int d = after > before ? 1 : -1;
    // up: the first entry from q + 2 on of at most `bound`; down: the first from q + 1 back, and
    // one more
    auto reach = [&](int bound) {
      int p = q + 2;
#pragma unroll
      for (int lv = kBuildLevels - 1; lv >= 0; --lv) {
        const int step = d * (1 << lv);
        if (least(lv, max(p + min(step, 0), 0)) > bound) p += step;
      }
      return p;
    };
    const int end = reach(min(before, after));
    if (after == before || end == (d > 0 ? kBuildEnd : 1)) {
      s_list[atomicAdd(&s_count, 1)] = (uint16_t)q;
      continue;
    }
    // the range's entries are [a, b): its smallest prefix is where it splits
    const int a = min(q + 2, end), b = max(q + 2, end);
    const int lv = 31 - __clz(b - a);
    const int split = reach(min(least(lv, a), least(lv, b - (1 << lv))));
    out.node(i, n, t0 - 2 + a, t0 - 2 + b, t0 - 2 + split + min(d, 0));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, part = lane & 7, group = threadIdx.x >> 3;
  const auto digits = [](int x) { return (31 - __clz(x)) / 3 * 3; };  // 8 << digits exceeds x
  for (int e0 = group & ~3; e0 < s_count; e0 += kBuildThreads / 8) {  // the same for the warp
    const int e = e0 + (group & 3), i = t0 + s_list[min(e, s_count - 1)];
    const int d = lcp(i, i + 1) > lcp(i, i - 1) ? 1 : -1;
    // how many of the lanes' distances, which rise, still have a prefix above `bound`
    auto within = [&](long long distance, int bound) {
      const long long j = i + d * distance;
      const bool in = j >= 0 && j < n && lcp(i, (int)j) > bound;
      const uint32_t past = ~__ballot_sync(0xffffffffu, in) >> (lane & 24) & 0xffu;
      return past ? __ffs(past) - 1 : 8;
    };
    // the largest such distance, an octal digit at a time
    auto reach = [&](int bound, int top) {
      int l = 0;
      for (int shift = __reduce_max_sync(0xffffffffu, top); shift >= 0; shift -= 3)
        l += max(within(l + ((long long)part << shift), bound) - 1, 0) << shift;
      return l;
    };
    const int outside = lcp(i, i - d), c = within(1ll << 3 * part, outside);
    const int l = reach(outside, c < 8 ? 3 * c - 3 : digits(n)), j = i + d * l;
    // (the split lies inside the range, whatever unsorted codes say)
    const int at = min(reach(lcp(i, j), digits(max(l, 1))), max(l - 1, 0));
    const int split = i + d * at + min(d, 0);
    if (part == 0 && e < s_count) out.node(i, n, min(i, j), max(i, j), split);
  }
}

// A thread per node, searching the codes.
template <class Lcp>
__global__ void __launch_bounds__(256) build_few_kernel(Lcp lcp, int n, ar_lbvh::TreeOut out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) out.parent[n] = -1;
  if (i < n - 1) ar_lbvh::karras_node(i, n, lcp, out);
}

// The tiles' barriers and the nodes that leave them cost a small tree more than the searches do.
// Where the two forms meet depends on the codes (kernels alone, searches against tiles: 30 spread
// bits 100,000 points 10.4 / 11.5 us, 150,000 11.1 / 11.5, 200,000 11.6 / 11.9, 262,144 13.9 /
// 12.3; 30 clustered bits 100,000 10.9 / 10.8, 150,000 12.1 / 11.2; 63 spread bits 100,000 11.9 /
// 12.1, 131,072 12.8 / 11.9, 200,000 13.4 / 12.6): the line lies between.
constexpr int kBuildTilesFrom = 1 << 17;
template <class Lcp>
void launch_build(const Lcp& lcp, int n, const ar_lbvh::TreeOut& out, cudaStream_t st) {
  if (n < kBuildTilesFrom)
    build_few_kernel<<<arh::grid_for(n - 1, 256), 256, 0, st>>>(lcp, n, out);
  else
    build_kernel<<<arh::grid_for(n - 1, kBuildTile), kBuildThreads, 0, st>>>(lcp, n, out);
}

// ---- leaves (kernelConstructLeafNodesSoA + initializeRadii, BVHSoAKernels.cu:108-138) ------
__global__ void __launch_bounds__(256) leaves_kernel(int n, const int32_t* __restrict__ sorted_idx,
                                                     const float4* __restrict__ pos, float r,
                                                     uint8_t* __restrict__ is_leaf,
                                                     int32_t* __restrict__ min_r,
                                                     int32_t* __restrict__ max_r,
                                                     float4* __restrict__ cms,
                                                     float4* __restrict__ bounds,
                                                     float* __restrict__ radii) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 c = __ldg(pos + __ldg(sorted_idx + i));
  is_leaf[i] = 1;
  min_r[i] = i;
  max_r[i] = i;
  cms[i] = c;
  bounds[2 * i] = make_float4(c.x - r, c.y - r, c.z - r, c.x + r);
  bounds[2 * i + 1] = make_float4(c.y + r, c.z + r, 0.f, 0.f);
  radii[i] = r;
}

// ---- refit (kernelConstructInternalNodesSoA, BVHSoAKernels.cu:148-176) ----------------------
// One thread per leaf climbs (ar_lbvh::refit_climb): the better form while the launch, and not the
// number of arrivals, bounds it.
__global__ void __launch_bounds__(256) refit_kernel(int n, const int32_t* __restrict__ left,
                                                    const int32_t* __restrict__ right,
                                                    const int32_t* __restrict__ parent,
                                                    float4* bounds, int* counters) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ar_lbvh::refit_climb(i, n, left, right, parent, bounds, counters);
}

// From this many leaves on the tiles below pay for their second launch (both forms: 400,000 points
// 57.8 us alone, 65.2 in tiles; 600,000: 67.5, 70.7; 800,000: 77.6, 80.4; 900,000: 85.0, 83.0;
// 1,000,003: 90.9, 87.6; 2,000,000: 150, 124).
constexpr int kRefitTilesFrom = 7 << 17;
// A block takes kRefitTile consecutive leaves and the internal nodes of the same numbers.  The
// subtrees that lie within these are merged in shared memory, the second child to arrive at a node
// merging both.  The largest of them are left to refit_open_kernel, which climbs the rest of the
// tree through global memory with ar_lbvh::refit_climb: a block that climbed on by itself would
// keep its place on the SM for its longest climb (2^24 points: 1006 us, without the prefetched
// links).  Any tree is refitted;
// Karras' numbering, which gives a node the number of one end of its leaves, makes all but about
// one node in twenty-five merge in shared memory, where a climb of every leaf through device-scope
// arrivals was bound by these (2^24 points: 953 -> 691 us).
// A subtree left over is named in the counter of a merged node, which nothing arrives at, as
// -(its root + 1); a tile with more of them than merged nodes climbs from the rest itself.
constexpr int kRefitTile = 256;
__global__ void __launch_bounds__(kRefitTile) refit_tiles_kernel(int n, const int32_t* __restrict__ left,
                                                           const int32_t* __restrict__ right,
                                                           const int32_t* __restrict__ parent,
                                                           float4* bounds,
                                                           int* __restrict__ counters) {
  constexpr int kT = kRefitTile;
  __shared__ float4 s_a[2 * kT], s_b[2 * kT];  // boxes: the tile's leaves, then its nodes
  __shared__ short s_child[2][kT];             // places of a node's children, -1: elsewhere
  __shared__ short s_parent[2 * kT];           // node of the tile above a place, -1: elsewhere
  __shared__ int s_met[kT];                    // children that have arrived
  __shared__ short s_slot[kT];                 // the merged nodes
  __shared__ int s_slots, s_open;
  const int t = threadIdx.x, base = blockIdx.x * kT, k = base + t;
  auto place = [&](int c) {
    const unsigned leaf = (unsigned)(c - base), node = (unsigned)(c - n - base);
    if (c < n) return leaf < (unsigned)kT ? (int)leaf : -1;
    return node < (unsigned)kT ? kT + (int)node : -1;
  };
  if (k < n) {
    s_a[t] = __ldcs(bounds + 2 * k);
    s_b[t] = __ldcs(bounds + 2 * k + 1);
  }
  int lc = -1, rc = -1;
  if (k < n - 1) {
    lc = place(__ldg(left + n + k));
    rc = place(__ldg(right + n + k));
  }
  s_child[0][t] = (short)lc;
  s_child[1][t] = (short)rc;
  s_parent[t] = s_parent[kT + t] = -1;
  s_met[t] = 0;
  if (t == 0) s_slots = s_open = 0;
  __syncthreads();
  if (lc >= 0 && rc >= 0) s_parent[lc] = s_parent[rc] = (short)t;
  __syncthreads();
  if (k < n) {
    int c = t, p = s_parent[t];
    float4 a = s_a[t], b = s_b[t];
    for (int guard = 0; guard < kT && p >= 0; ++guard, p = s_parent[c]) {
      __threadfence_block();  // this child's box before its arrival
      if (atomicAdd(&s_met[p], 1) != 1) break;
      __threadfence_block();  // its sibling's box after that one's arrival
      const bool is_left = s_child[0][p] == c;
      const int o = s_child[is_left ? 1 : 0][p];
      const float4 oa = s_a[o], ob = s_b[o];
      const ar_lbvh::Box6 u = is_left ? ar_lbvh::merge_boxes(ar_lbvh::box6(a, b), ar_lbvh::box6(oa, ob))
                                      : ar_lbvh::merge_boxes(ar_lbvh::box6(oa, ob), ar_lbvh::box6(a, b));
      c = kT + p;
      a = s_a[c] = make_float4(u.lx, u.ly, u.lz, u.hx);
      b = s_b[c] = make_float4(u.hy, u.hz, 0.f, 0.f);
    }
  }
  __syncthreads();
  // the merged nodes' boxes; the leaves and merged nodes whose parent is not merged are left over
  const bool merged = s_met[t] >= 2;
  if (merged) {
    __stcg(bounds + 2 * (size_t)(n + k), s_a[kT + t]);
    __stcg(bounds + 2 * (size_t)(n + k) + 1, s_b[kT + t]);
  }
  auto open = [&](int c) { return s_parent[c] < 0 || s_met[s_parent[c]] < 2; };
  const bool open_leaf = k < n && open(t), open_node = merged && open(kT + t);
  if (merged) s_slot[atomicAdd(&s_slots, 1)] = (short)t;
  const int at = open_leaf || open_node ? atomicAdd(&s_open, (int)open_leaf + (int)open_node) : 0;
  __syncthreads();
  auto leave = [&](int root, int i) {
    if (i < s_slots) counters[base + s_slot[i]] = -(root + 1);
    else ar_lbvh::refit_climb(root, n, left, right, parent, bounds, counters);
  };
  if (open_leaf) leave(k, at);
  if (open_node) leave(n + k, at + (int)open_leaf);
}

// The climb from the subtrees that refit_tiles_kernel left over: a block collects those of kRefitScan
// counters, so that its threads climb together.
constexpr int kRefitScan = 4096;
__global__ void __launch_bounds__(256) refit_open_kernel(int n, const int32_t* __restrict__ left,
                                                         const int32_t* __restrict__ right,
                                                         const int32_t* __restrict__ parent,
                                                         float4* bounds, int* counters) {
  __shared__ int s_root[kRefitScan];
  __shared__ int s_count;
  if (threadIdx.x == 0) s_count = 0;
  __syncthreads();
  const long base = (long)blockIdx.x * kRefitScan;
  for (int i = threadIdx.x; i < kRefitScan; i += blockDim.x) {
    const int v = base + i < n - 1 ? __ldcg(counters + base + i) : 0;
    if (v < 0) s_root[atomicAdd(&s_count, 1)] = -v - 1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < s_count; i += blockDim.x)
    ar_lbvh::refit_climb(s_root[i], n, left, right, parent, bounds, counters);
}

// Parent links from the child links, for callers with the reference's traversal signature
// (collideBVHSoARigidBodyWrapper passes no parent array): one thread per internal node.
__global__ void __launch_bounds__(256) parents_kernel(int n, const int32_t* __restrict__ left,
                                                      const int32_t* __restrict__ right,
                                                      int32_t* __restrict__ parent) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int node = n + i;
  parent[__ldg(left + node)] = node;
  parent[__ldg(right + node)] = node;
  if (i == 0) parent[n] = -1;
}

// ---- collideBVHSoARigidBody (Kernels/RB_BVHKernels.cu:100-244) ------------------------------
__global__ void __launch_bounds__(128) collide_bvh_kernel(
    ar_sim_params prm, const int32_t* __restrict__ rb_idx, const float4* __restrict__ rel,
    const float4* __restrict__ vel, const int32_t* __restrict__ left,
    const int32_t* __restrict__ right,
    const int32_t* __restrict__ parent, const float4* __restrict__ cms,
    const float4* __restrict__ bounds, const int32_t* __restrict__ sorted_idx,
    const float* __restrict__ radii, int n, float4* __restrict__ p_force,
    float4* __restrict__ p_torque, float4* __restrict__ p_positions) {
  const int index = blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= n) return;
  const int q = __ldg(sorted_idx + index);
  const float3 qvel = ar::xyz(__ldg(vel + q));
  const float4 qpos = __ldg(cms + index);
  const float qrad = __ldg(radii + index);
  const int qbody = __ldg(rb_idx + q);
  const Box qbox = load_box(bounds, index);
  const float4 qrel = __ldg(rel + q);
  const float4 rbcm = make_float4(qpos.x - qrel.x, qpos.y - qrel.y, qpos.z - qrel.z, qpos.w - qrel.w);
  float3 force = ar::mk3(0.f, 0.f, 0.f), torque = ar::mk3(0.f, 0.f, 0.f);
  float4 corr = make_float4(0.f, 0.f, 0.f, 0.f);
  const float3 r3 = ar::xyz(qrel);
  if (n >= 2) {
    ar_lbvh::walk(n, n, left, right, parent,
         [&](int c) { return c != index && overlap(qbox, load_box(bounds, c)); },
         [&](int c, bool is_left) {
           const int oc = __ldg(sorted_idx + c);
           const int ob = __ldg(rb_idx + oc);
           if (!(qbody != ob || qbody == -1)) return;
           float4 lc = make_float4(0.f, 0.f, 0.f, 0.f);
           float3 f = ar_dem::static_pair(qpos, __ldg(cms + c), rbcm, qvel,
                                          ar::xyz(__ldg(vel + oc)), qrad, __ldg(radii + c), prm,
                                          &lc);
           if (!is_left) {  // the right-leaf branch also takes maxOpF4(local, corr) first (:191)
             corr.x = corr.x > lc.x ? corr.x : lc.x;
             corr.y = corr.y > lc.y ? corr.y : lc.y;
             corr.z = corr.z > lc.z ? corr.z : lc.z;
             corr.w = corr.w > lc.w ? corr.w : lc.w;
           }
           corr = make_float4(corr.x + lc.x, corr.y + lc.y, corr.z + lc.z, corr.w + lc.w);
           force = ar::add(force, f);
           torque = ar::add(torque, ar::cross(r3, f));
         });
  }
  if (qbody == -1) return;  // free particles: the reference updates vel in place (not on this path)
  p_force[q] = make_float4(force.x, force.y, force.z, 0.f);
  p_torque[q] = make_float4(torque.x, torque.y, torque.z, 0.f);
  if (p_positions) p_positions[q] = corr;
}

// ---- FindRigidBodyCollisionsBVHKernel (Kernels/RB_BVHKernels.cu:760-876) ---------------------
__global__ void __launch_bounds__(128) find_contacts_kernel(
    const int32_t* __restrict__ rb_idx, const int32_t* __restrict__ left,
    const int32_t* __restrict__ right,
    const int32_t* __restrict__ parent, const int32_t* __restrict__ max_r,
    const float4* __restrict__ cms, const float4* __restrict__ bounds,
    const int32_t* __restrict__ sorted_idx, const float* __restrict__ radii, int n,
    float* __restrict__ contact_distance, int32_t* __restrict__ colliding_particle,
    int32_t* __restrict__ colliding_body) {
  const int index = blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= n || n < 2) return;
  const int q = __ldg(sorted_idx + index);
  const float4 qpos = __ldg(cms + index);
  const Box qbox = load_box(bounds, index);
  const float qrad = __ldg(radii + q);
  const int qbody = __ldg(rb_idx + q);
  float best = contact_distance[q];
  int best_p = 0, best_b = 0;
  bool found = false;
  ar_lbvh::walk(n, n, left, right, parent,
       [&](int c) {
         return c != index && __ldg(max_r + c) >= index && overlap(qbox, load_box(bounds, c));
       },
       [&](int c, bool) {
         const int oc = __ldg(sorted_idx + c);
         const int ob = __ldg(rb_idx + oc);
         if (qbody == ob) return;
         const float4 cp = __ldg(cms + c);
         const float4 dd = make_float4(cp.x - qpos.x, cp.y - qpos.y, cp.z - qpos.z, cp.w - qpos.w);
         const float dist = sqrtf(dd.x * dd.x + dd.y * dd.y + dd.z * dd.z + dd.w * dd.w);
         const float thr = qrad + __ldg(radii + oc);
         if (thr - dist > best) {
           best = thr - dist;
           best_p = oc;
           best_b = ob;
           found = true;
         }
       });
  if (found) {
    contact_distance[q] = best;
    colliding_particle[q] = best_p;
    colliding_body[q] = best_b;
  }
}

// ---- contact pairs through the BVH ------------------------------------------------------------
__global__ void __launch_bounds__(128) pairs_bvh_kernel(
    float two_r, const int32_t* __restrict__ rb_idx, const int32_t* __restrict__ left,
    const int32_t* __restrict__ right,
    const int32_t* __restrict__ parent, const float4* __restrict__ cms,
    const float4* __restrict__ bounds, const int32_t* __restrict__ sorted_idx, int n,
    int2* __restrict__ pairs, int capacity, int* __restrict__ count, int* __restrict__ err) {
  const int index = blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= n || n < 2) return;
  const int q = __ldg(sorted_idx + index);
  const float4 qpos = __ldg(cms + index);
  const Box qbox = load_box(bounds, index);
  const int qbody = __ldg(rb_idx + q);
  ar_lbvh::walk(n, n, left, right, parent,
       [&](int c) { return c != index && overlap(qbox, load_box(bounds, c)); },
       [&](int c, bool) {
         if (c < index) return;  // each unordered pair once (from its lower sorted leaf)
         const int oc = __ldg(sorted_idx + c);
         if (__ldg(rb_idx + oc) == qbody) return;
         if (!ar_dem::touching(ar::xyz(qpos), ar::xyz(__ldg(cms + c)), two_r)) return;
         int slot = atomicAdd(count, 1);
         if (slot < capacity)
           pairs[slot] = make_int2(min(q, oc), max(q, oc));
         else
           ar::raise_error(err, ar::kErrOverflow);
       });
}


// ---- static scene through a BVH over its point cloud ----------------------------------------
// checkOverlap(float4, AABB, radius) (BVHSource/BVHAuxiliary.cuh:159-175): the box point
// closest to the sphere centre, distance rounded toward zero, strictly below the radius.
__device__ __forceinline__ bool sphere_box(float4 p, const Box& b, float r) {
  const float xx = fmaxf(b.lx, fminf(p.x, b.hx));
  const float yy = fmaxf(b.ly, fminf(p.y, b.hy));
  const float zz = fmaxf(b.lz, fminf(p.z, b.hz));
  const float d = __fsqrt_rz((xx - p.x) * (xx - p.x) + (yy - p.y) * (yy - p.y) +
                             (zz - p.z) * (zz - p.z));
  return d < r;
}

// staticCollideBVHSoARigidBody (Kernels/RB_BVHKernels.cu:293-442): particle i (unsorted, radius
// params.particle_radius) walks the scene's tree (m leaves) in the reference's order; every
// overlapping leaf adds the DEM force of collideSpheresBVH (BVHAuxiliary.cuh:97-130, the scene
// point at rest) and rel x force.  The reference adds a body's particles' totals straight into
// the body's force and torque with plain read-modify-writes from many threads (racy); here each
// particle's totals go to p_force4 / p_torque4 at its index, for a fixed-order body sum
// (ar_reduce_bodies).  A free particle (body -1) gets v + force as its velocity.  color4 (may
// be NULL): green when a leaf is within touching distance.
__global__ void __launch_bounds__(128) collide_bvh_static_kernel(
    ar_sim_params prm, const int32_t* __restrict__ rb_idx, const float4* __restrict__ rel,
    const float4* __restrict__ pos, float4* __restrict__ vel, const int32_t* __restrict__ left,
    const int32_t* __restrict__ right,
    const int32_t* __restrict__ parent, const float4* __restrict__ cms,
    const float4* __restrict__ bounds, const float* __restrict__ radii, int m, int n,
    float4* __restrict__ p_force, float4* __restrict__ p_torque, float4* __restrict__ color) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 qpos = __ldg(pos + i);
    const float3 qvel = ar::xyz(vel[i]);
    const float qrad = prm.particle_radius;
    const int qbody = __ldg(rb_idx + i);
    const float3 r3 = ar::xyz(__ldg(rel + i));
    float3 force = ar::mk3(0.f, 0.f, 0.f), torque = force;
    if (m >= 2) {
      ar_lbvh::walk(m, m, left, right, parent,
                    [&](int c) { return sphere_box(qpos, load_box(bounds, c), qrad); },
                    [&](int c, bool) {
                      const float4 cp = __ldg(cms + c);
                      const float rc = __ldg(radii + c);
                      const float3 rp = ar::mk3(cp.x - qpos.x, cp.y - qpos.y, cp.z - qpos.z);
                      const float dist = sqrtf(ar::dot(rp, rp));
                      float3 f = ar::mk3(0.f, 0.f, 0.f);
                      if (dist < qrad + rc)
                        f = ar_dem::spring_force(rp, dist,
                                                 ar::mk3(0.f - qvel.x, 0.f - qvel.y, 0.f - qvel.z),
                                                 qrad + rc, prm.spring, prm.damping, prm.shear,
                                                 prm.attraction);
                      force = ar::add(force, f);
                      torque = ar::add(torque, ar::cross(r3, f));
                      if (dist < qrad + rc && color) color[i] = make_float4(0.f, 1.f, 0.f, 0.f);
                    });
    }
    if (qbody >= 0) {
      p_force[i] = make_float4(force.x, force.y, force.z, 0.f);
      p_torque[i] = make_float4(torque.x, torque.y, torque.z, 0.f);
    } else {
      vel[i] = make_float4(qvel.x + force.x, qvel.y + force.y, qvel.z + force.z, 0.f);
    }
  }
}

// FindAugmentedRealityCollisionsBVHKernel (Kernels/RB_BVHKernels.cu:920-1023): deepest contact
// of particle i with the scene through its tree: an overlapping leaf c (cloud point
// sorted_idx[c]) deepens the contact when r + radii[point] - |cms[c] - p| (four components, as
// the reference's length(float4)) exceeds contact_distance[i], which records it with the point.
// The query radius is params.particle_radius (the reference reads the scene's radius array at
// the query's index; the two agree when every radius is the particle radius).  color4 (may be
// NULL): green on a contact, white when none.
__global__ void __launch_bounds__(128) find_bvh_static_kernel(
    ar_sim_params prm, const float4* __restrict__ pos, const int32_t* __restrict__ left,
    const int32_t* __restrict__ right,
    const int32_t* __restrict__ parent, const float4* __restrict__ cms,
    const float4* __restrict__ bounds, const int32_t* __restrict__ sorted_idx,
    const float* __restrict__ radii, int m, int n, float* __restrict__ contact_distance,
    int32_t* __restrict__ contact_point, float4* __restrict__ color) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 qpos = __ldg(pos + i);
    const float qrad = prm.particle_radius;
    float deepest = contact_distance[i];
    int best = contact_point[i], ncol = 0;
    if (m >= 2) {
      ar_lbvh::walk(m, m, left, right, parent,
                    [&](int c) { return sphere_box(qpos, load_box(bounds, c), qrad); },
                    [&](int c, bool) {
                      const int s = __ldg(sorted_idx + c);
                      const float4 cp = __ldg(cms + c);
                      const float4 d = make_float4(cp.x - qpos.x, cp.y - qpos.y, cp.z - qpos.z,
                                                   cp.w - qpos.w);
                      const float dist = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w);
                      const float thr = qrad + __ldg(radii + s);
                      if (thr - dist > deepest) {
                        ++ncol;
                        deepest = thr - dist;
                        best = s;
                      }
                    });
    }
    contact_distance[i] = deepest;
    contact_point[i] = best;
    if (color) color[i] = ncol ? make_float4(0.f, 1.f, 0.f, 0.f) : make_float4(1.f, 1.f, 1.f, 0.f);
  }
}

// parent links: the caller's, or derived into scratch when the caller has none
const int32_t* parents_or_derive(ar_ctx* ctx, int n, const int32_t* left, const int32_t* right,
                                 const int32_t* parent, cudaStream_t st) {
  if (parent || n < 2) return parent;
  int32_t* p = (int32_t*)arh::scratch(ctx, (size_t)(2 * n - 1) * sizeof(int32_t));
  if (!p) return nullptr;
  parents_kernel<<<arh::grid_for(n - 1, 256), 256, 0, st>>>(n, left, right, p);
  return p;
}

}  // namespace

extern "C" {

ar_status ar_lbvh_build(ar_ctx* ctx, const uint32_t* sorted_codes, int n, uint8_t* is_leaf,
                        int32_t* left, int32_t* right, int32_t* parent, int32_t* min_r,
                        int32_t* max_r, ar_stream_t stream) {
  if (!ctx || n < 0 || (n > 0 && (!sorted_codes || !is_leaf || !left || !right || !parent ||
                                  !min_r || !max_r)))
    return AR_ERR_INVALID_ARG;
  if (n < 2) return AR_OK;
  launch_build(ar_lbvh::Lcp32{sorted_codes, n}, n,
               ar_lbvh::TreeOut{is_leaf, left, right, parent, min_r, max_r}, arh::stream(stream));
  return arh::check_launch("ar_lbvh_build");
}

ar_status ar_lbvh_build64(ar_ctx* ctx, const uint64_t* sorted_codes, int n, uint8_t* is_leaf,
                          int32_t* left, int32_t* right, int32_t* parent, int32_t* min_r,
                          int32_t* max_r, ar_stream_t stream) {
  if (!ctx || n < 0 || (n > 0 && (!sorted_codes || !is_leaf || !left || !right || !parent ||
                                  !min_r || !max_r)))
    return AR_ERR_INVALID_ARG;
  if (n < 2) return AR_OK;
  launch_build(ar_lbvh::Lcp64{sorted_codes, n}, n,
               ar_lbvh::TreeOut{is_leaf, left, right, parent, min_r, max_r}, arh::stream(stream));
  return arh::check_launch("ar_lbvh_build64");
}

ar_status ar_lbvh_leaves(ar_ctx* ctx, int n, const int32_t* sorted_idx, const float* pos4,
                         float radius, uint8_t* is_leaf, int32_t* min_r, int32_t* max_r,
                         float* cms4, float* bounds8, float* radii, ar_stream_t stream) {
  if (!ctx || n < 0 ||
      (n > 0 && (!sorted_idx || !pos4 || !is_leaf || !min_r || !max_r || !cms4 || !bounds8 ||
                 !radii)))
    return AR_ERR_INVALID_ARG;
  if (n == 0) return AR_OK;
  leaves_kernel<<<arh::grid_for(n, 256), 256, 0, arh::stream(stream)>>>(
      n, sorted_idx, (const float4*)pos4, radius, is_leaf, min_r, max_r, (float4*)cms4,
      (float4*)bounds8, radii);
  return arh::check_launch("ar_lbvh_leaves");
}

ar_status ar_lbvh_refit(ar_ctx* ctx, int n, const int32_t* left, const int32_t* right,
                        const int32_t* parent, float* bounds8, ar_stream_t stream) {
  if (!ctx || n < 0 || (n > 0 && (!left || !right || !parent || !bounds8)))
    return AR_ERR_INVALID_ARG;
  if (n < 2) return AR_OK;
  int* counters = (int*)arh::scratch(ctx, (size_t)(n - 1) * sizeof(int));
  if (!counters) return AR_ERR_OOM;
  cudaStream_t st = arh::stream(stream);
  cudaMemsetAsync(counters, 0, (size_t)(n - 1) * sizeof(int), st);
  if (n < kRefitTilesFrom) {
    refit_kernel<<<arh::grid_for(n, 256), 256, 0, st>>>(n, left, right, parent, (float4*)bounds8,
                                                        counters);
  } else {
    refit_tiles_kernel<<<arh::grid_for(n, kRefitTile), kRefitTile, 0, st>>>(
        n, left, right, parent, (float4*)bounds8, counters);
    refit_open_kernel<<<arh::grid_for(n - 1, kRefitScan), 256, 0, st>>>(
        n, left, right, parent, (float4*)bounds8, counters);
  }
  return arh::check_launch("ar_lbvh_refit");
}

ar_status ar_collide_bvh_dem(ar_ctx* ctx, const ar_sim_params* params, const int32_t* rb_idx,
                             const float* rel4, const float* vel4, const uint8_t* is_leaf,
                             const int32_t* left, const int32_t* right, const int32_t* parent,
                             const float* cms4, const float* bounds8, const int32_t* sorted_idx,
                             const float* radii, int n, float* p_force4, float* p_torque4,
                             float* p_positions4, ar_stream_t stream) {
  if (!ctx || !params || n < 0 ||
      (n > 0 && (!rb_idx || !rel4 || !vel4 || !is_leaf || !left || !right ||
                 !cms4 || !bounds8 || !sorted_idx || !radii || !p_force4 || !p_torque4)))
    return AR_ERR_INVALID_ARG;
  if (n == 0) return AR_OK;
  parent = parents_or_derive(ctx, n, left, right, parent, arh::stream(stream));
  if (!parent && n >= 2) return AR_ERR_OOM;
  collide_bvh_kernel<<<arh::grid_for(n, 128), 128, 0, arh::stream(stream)>>>(
      *params, rb_idx, (const float4*)rel4, (const float4*)vel4, left, right, parent,
      (const float4*)cms4, (const float4*)bounds8, sorted_idx, radii, n, (float4*)p_force4,
      (float4*)p_torque4, (float4*)p_positions4);
  return arh::check_launch("ar_collide_bvh_dem");
}

ar_status ar_collide_bvh_static(ar_ctx* ctx, const ar_sim_params* params, const int32_t* rb_idx,
                                const float* rel4, const float* pos4, float* vel4,
                                const uint8_t* is_leaf, const int32_t* left,
                                const int32_t* right, const int32_t* parent, const float* cms4,
                                const float* bounds8, const float* radii, int num_scene, int n,
                                float* p_force4, float* p_torque4, float* color4,
                                ar_stream_t stream) {
  if (!ctx || !params || n < 0 || num_scene < 0 ||
      (n > 0 && (!rb_idx || !rel4 || !pos4 || !vel4 || !p_force4 || !p_torque4)) ||
      (num_scene >= 2 && (!is_leaf || !left || !right || !cms4 || !bounds8 || !radii)))
    return AR_ERR_INVALID_ARG;
  if (n == 0) return AR_OK;
  cudaStream_t st = arh::stream(stream);
  parent = parents_or_derive(ctx, num_scene, left, right, parent, st);
  if (!parent && num_scene >= 2) return AR_ERR_OOM;
  const unsigned grid = std::min(arh::grid_for(n, 128), (unsigned)ctx->num_sms * 16);
  collide_bvh_static_kernel<<<grid, 128, 0, st>>>(
      *params, rb_idx, (const float4*)rel4, (const float4*)pos4, (float4*)vel4, left,
      right, parent, (const float4*)cms4, (const float4*)bounds8, radii, num_scene, n,
      (float4*)p_force4, (float4*)p_torque4, (float4*)color4);
  return arh::check_launch("ar_collide_bvh_static");
}

ar_status ar_find_contacts_bvh_static(ar_ctx* ctx, const ar_sim_params* params,
                                      const float* pos4, const uint8_t* is_leaf,
                                      const int32_t* left, const int32_t* right,
                                      const int32_t* parent, const float* cms4,
                                      const float* bounds8, const int32_t* sorted_idx,
                                      const float* radii, int num_scene, int n,
                                      float* contact_distance, int32_t* contact_point,
                                      float* color4, ar_stream_t stream) {
  if (!ctx || !params || n < 0 || num_scene < 0 ||
      (n > 0 && (!pos4 || !contact_distance || !contact_point)) ||
      (num_scene >= 2 && (!is_leaf || !left || !right || !cms4 || !bounds8 || !sorted_idx ||
                          !radii)))
    return AR_ERR_INVALID_ARG;
  if (n == 0) return AR_OK;
  cudaStream_t st = arh::stream(stream);
  parent = parents_or_derive(ctx, num_scene, left, right, parent, st);
  if (!parent && num_scene >= 2) return AR_ERR_OOM;
  const unsigned grid = std::min(arh::grid_for(n, 128), (unsigned)ctx->num_sms * 16);
  find_bvh_static_kernel<<<grid, 128, 0, st>>>(
      *params, (const float4*)pos4, left, right, parent, (const float4*)cms4,
      (const float4*)bounds8, sorted_idx, radii, num_scene, n, contact_distance, contact_point,
      (float4*)color4);
  return arh::check_launch("ar_find_contacts_bvh_static");
}

ar_status ar_find_contacts_bvh(ar_ctx* ctx, const int32_t* rb_idx, const uint8_t* is_leaf,
                               const int32_t* left, const int32_t* right, const int32_t* parent,
                               const int32_t* max_r, const float* cms4, const float* bounds8,
                               const int32_t* sorted_idx, const float* radii, int n,
                               float* contact_distance, int32_t* colliding_particle,
                               int32_t* colliding_body, ar_stream_t stream) {
  if (!ctx || n < 0 ||
      (n > 0 && (!rb_idx || !is_leaf || !left || !right || !max_r || !cms4 ||
                 !bounds8 || !sorted_idx || !radii || !contact_distance ||
                 !colliding_particle || !colliding_body)))
    return AR_ERR_INVALID_ARG;
  if (n < 2) return AR_OK;
  parent = parents_or_derive(ctx, n, left, right, parent, arh::stream(stream));
  if (!parent) return AR_ERR_OOM;
  find_contacts_kernel<<<arh::grid_for(n, 128), 128, 0, arh::stream(stream)>>>(
      rb_idx, left, right, parent, max_r, (const float4*)cms4, (const float4*)bounds8,
      sorted_idx, radii, n, contact_distance, colliding_particle, colliding_body);
  return arh::check_launch("ar_find_contacts_bvh");
}

ar_status ar_pairs_bvh(ar_ctx* ctx, float radius, const int32_t* rb_idx, const uint8_t* is_leaf,
                       const int32_t* left, const int32_t* right, const int32_t* parent,
                       const float* cms4, const float* bounds8, const int32_t* sorted_idx, int n,
                       int32_t* pairs2, int capacity, int32_t* d_count, ar_stream_t stream) {
  if (!ctx || n < 0 || capacity < 0 || !d_count ||
      (n > 0 && (!rb_idx || !is_leaf || !left || !right || !cms4 || !bounds8 ||
                 !sorted_idx || (capacity > 0 && !pairs2))))
    return AR_ERR_INVALID_ARG;
  cudaStream_t st = arh::stream(stream);
  cudaMemsetAsync(d_count, 0, sizeof(int32_t), st);
  if (n < 2) return arh::check_launch("ar_pairs_bvh");
  parent = parents_or_derive(ctx, n, left, right, parent, st);
  if (!parent) return AR_ERR_OOM;
  pairs_bvh_kernel<<<arh::grid_for(n, 128), 128, 0, st>>>(
      2.0f * radius, rb_idx, left, right, parent, (const float4*)cms4,
      (const float4*)bounds8, sorted_idx, n, (int2*)pairs2, capacity, d_count, ctx->d_err);
  return arh::check_launch("ar_pairs_bvh");
}

}  // extern "C"
