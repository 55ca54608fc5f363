// LBVH device routines shared by the stage entry points (ar_lbvh.cu) and the fused BVH step
// (ar_pipeline.cu): Karras node construction, fenced bottom-up refit, box tests and the
// traversal in the reference's visit order.
//
// Node numbering is the reference's SoA layout (BVHSource/BVHSoAKernels.cu): leaf i at index
// i, internal node i at n + i, root at n.  Boxes are the reference's 32-byte AABB
// {min.xyz, max.xyz, pad, pad}, read as two float4.
#pragma once
#include <cuda/atomic>

#include "ar_internal.cuh"

namespace ar_lbvh {

// ---- longest common prefix (BVHSource/BVHAuxiliary.cuh:31-43) ------------------------------
struct Lcp32 {
  const uint32_t* __restrict__ c;
  int n;
  __device__ __forceinline__ int operator()(int i, int j) const {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = __ldg(c + i), b = __ldg(c + j);
    return a != b ? __clz(a ^ b) : __clz(i ^ j) + 32;
  }
};
struct Lcp64 {
  const uint64_t* __restrict__ c;
  int n;
  __device__ __forceinline__ int operator()(int i, int j) const {
    if (j < 0 || j >= n) return -1;
    const uint64_t a = __ldg((const unsigned long long*)c + i),
                   b = __ldg((const unsigned long long*)c + j);
    return a != b ? __clzll(a ^ b) : __clz(i ^ j) + 64;
  }
};
// 64-bit keys whose top bits (>> shift) name a scene: equal keys are tie-broken by their index
// within the scene, so a scene's subtree is the same as in a tree built over the scene alone.
struct Lcp64Scene {
  const uint64_t* __restrict__ c;
  int n;
  const int* __restrict__ poff;
  int shift;
  __device__ __forceinline__ int operator()(int i, int j) const {
    if (j < 0 || j >= n) return -1;
    const uint64_t a = __ldg((const unsigned long long*)c + i),
                   b = __ldg((const unsigned long long*)c + j);
    if (a != b) return __clzll(a ^ b);
    const int base = __ldg(poff + (int)(a >> shift));
    return __clz((i - base) ^ (j - base)) + 64;
  }
};

// The same for 32-bit keys (scene index above the 30-bit code, at most 4 scenes).  Its
// values are those of Lcp64Scene minus 32 for the same keys, so the topology is the same.
struct Lcp32Scene {
  const uint32_t* __restrict__ c;
  int n;
  const int* __restrict__ poff;
  int shift;
  __device__ __forceinline__ int operator()(int i, int j) const {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = __ldg(c + i), b = __ldg(c + j);
    if (a != b) return __clz(a ^ b);
    const int base = __ldg(poff + (int)(a >> shift));
    return __clz((i - base) ^ (j - base)) + 32;
  }
};

// ---- Karras 2012 internal nodes (kernelConstructRadixTreeSoA, BVHSoAKernels.cu:7-99) ----
struct TreeOut {
  uint8_t* is_leaf;
  int32_t *left, *right, *parent, *min_r, *max_r;
  // Internal node i over the leaves [lo, hi], split after leaf gamma.
  __device__ __forceinline__ void node(int i, int n, int lo, int hi, int gamma) const {
    const int node = n + i;
    is_leaf[node] = 0;
    const int lc = (lo == gamma) ? gamma : gamma + n;
    const int rc = (hi == gamma + 1) ? gamma + 1 : gamma + 1 + n;
    left[node] = lc;
    right[node] = rc;
    parent[lc] = node;
    parent[rc] = node;
    min_r[node] = lo;
    max_r[node] = hi;
  }
};

// Node i from the sorted codes alone.
template <class Lcp>
__device__ void karras_node(int i, int n, const Lcp& lcp, const TreeOut& out) {
  const int d = (lcp(i, i + 1) - lcp(i, i - 1)) > 0 ? 1 : -1;
  const int sig_min = lcp(i, i - d);
  int lmax = 2;
  while (lcp(i, i + lmax * d) > sig_min) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2) {
    if (lcp(i, i + (l + t) * d) > sig_min) l += t;
    if (t == 1) break;
  }
  const int j = i + l * d;
  const int sig_node = lcp(i, j);
  // split search: t = ceil(l / 2^k), k = 1, 2, ... (the reference's double division by a
  // power of two is exact, so the integer ceiling is the same value)
  int s = 0;
  for (int k = 1;; ++k) {
    const int t = (int)(((long long)l + (1ll << k) - 1) >> k);
    if (lcp(i, i + (s + t) * d) > sig_node) s += t;
    if (t <= 1) break;
  }
  out.node(i, n, min(i, j), max(i, j), i + s * d + min(d, 0));
}

// ---- bottom-up refit (kernelConstructInternalNodesSoA, BVHSoAKernels.cu:148-176) ------------
// The second thread to reach a node merges its children's boxes (mergeBounds,
// BVHAuxiliary.cuh:83-94: min of the mins and max of the maxes, left child first) and climbs on.
// The arrival counter is a device-scope acquire-release increment, so the first thread's box
// stores (made before its increment) are visible to the second thread's loads (made after it);
// boxes are read and written through L2.
struct Box6 {
  float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ Box6 merge_boxes(const Box6& a, const Box6& b) {  // a = left child
  return Box6{a.lx < b.lx ? a.lx : b.lx, a.ly < b.ly ? a.ly : b.ly, a.lz < b.lz ? a.lz : b.lz,
              a.hx > b.hx ? a.hx : b.hx, a.hy > b.hy ? a.hy : b.hy, a.hz > b.hz ? a.hz : b.hz};
}

// Returns the previous count.
__device__ __forceinline__ int arrive(int* counter) {
  cuda::atomic_ref<int, cuda::thread_scope_device> a(*counter);
  return a.fetch_add(1, cuda::memory_order_acq_rel);
}

__device__ __forceinline__ Box6 box6(const float4& a, const float4& b) {
  return Box6{a.x, a.y, a.z, a.w, b.x, b.y};
}
// Climb from `from`, a node whose box is final, merging and storing the boxes of the nodes at which
// this thread arrives second (two float4 per node).  A level costs two dependent round trips, the
// arrival and the sibling's box: the links of the next node are loaded with the box, and the
// child's own box is at hand.
__device__ __forceinline__ void refit_climb(int from, int n, const int32_t* __restrict__ left,
                                            const int32_t* __restrict__ right,
                                            const int32_t* __restrict__ parent, float4* bounds,
                                            int* counters) {
  // else the link is malformed, or there is no node
  auto inner = [&](int node) { return node >= n && node < 2 * n - 1; };
  int child = from, node = __ldg(parent + from);
  Box6 own = box6(__ldcg(bounds + 2 * (size_t)from), __ldcg(bounds + 2 * (size_t)from + 1));
  if (!inner(node)) return;
  int l = __ldg(left + node), r = __ldg(right + node), up = node != n ? __ldg(parent + node) : -1;
  for (int depth = 0; depth < n; ++depth) {  // a valid tree is at most n - 1 deep
    if (arrive(counters + (node - n)) == 0) return;
    const bool is_left = l == child;
    const float4* sib = bounds + 2 * (size_t)(is_left ? r : l);
    const float4 a = __ldcg(sib), b = __ldcg(sib + 1);
    int nl = -1, nr = -1, nup = -1;
    if (inner(up)) {
      nl = __ldg(left + up);
      nr = __ldg(right + up);
      if (up != n) nup = __ldg(parent + up);
    }
    own = is_left ? merge_boxes(own, box6(a, b)) : merge_boxes(box6(a, b), own);
    float4* to = bounds + 2 * (size_t)node;
    __stcg(to, make_float4(own.lx, own.ly, own.lz, own.hx));
    __stcg(to + 1, make_float4(own.hy, own.hz, 0.f, 0.f));
    if (!inner(up)) return;
    child = node;
    node = up;
    l = nl;
    r = nr;
    up = nup;
  }
}

// ---- boxes -----------------------------------------------------------------------------------
struct Box {
  float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ Box load_box(const float4* __restrict__ b, int node) {
  const float4 p = __ldg(b + 2 * node), q = __ldg(b + 2 * node + 1);
  return Box{p.x, p.y, p.z, p.w, q.x, q.y};
}
// checkOverlap(AABB, AABB) (BVHAuxiliary.cuh:139-152)
__device__ __forceinline__ bool overlap(const Box& a, const Box& b) {
  return (a.lx <= b.hx && a.hx >= b.lx) && (a.ly <= b.hy && a.hy >= b.ly) &&
         (a.lz <= b.hz && a.hz >= b.lz);
}

// ---- traversal in the reference's order (RB_BVHKernels.cu:145-214) ------------------------------
// From internal node `root`: at each internal node, the overlapping leaf children are handled
// left then right, then the walk descends into the left internal child if it overlaps, and on
// the way back up into the right one.  visit_leaf(leaf, is_left_child) for every leaf child
// that accept(child) admits (leaves are the nodes below n).  `root` is never left through its
// parent link.
//
// The right children to come back to wait on a short stack, the newest kStack of them: a tree
// over 32-bit keys rarely needs more.  Older ones are dropped, and found again once the stack is
// empty by climbing the parent links from the subtree just finished, so that no depth is too
// great.  Climbing after every subtree instead reads each node's links and boxes a second time on
// the way up (132,651 packed particles: 341 -> 175 us).  A valid tree is walked in fewer than
// 4 (2n - 1) moves; the bound only guards against a malformed tree.
constexpr int kStack = 32;  // a power of two
template <class Accept, class Visit>
__device__ __forceinline__ void walk(int root, int n, const int32_t* __restrict__ left,
                                     const int32_t* __restrict__ right,
                                     const int32_t* __restrict__ parent, Accept accept,
                                     Visit visit_leaf) {
  int stack[kStack];
  int top = 0, bottom = 0;  // entries bottom .. top - 1, at their index mod kStack
  int node = root, start = root;  // start: the root of the subtree being walked
  for (long moves = 8l * n + 64; moves > 0; --moves) {
    const int lc = __ldg(left + node), rc = __ldg(right + node);
    const bool ol = accept(lc), orr = accept(rc);
    if (ol && lc < n) visit_leaf(lc, true);
    if (orr && rc < n) visit_leaf(rc, false);
    const bool tl = ol && lc >= n, tr = orr && rc >= n;
    if (tl) {
      if (tr) {
        stack[top++ & (kStack - 1)] = rc;
        if (top - bottom > kStack) ++bottom;
      }
      node = lc;
      continue;
    }
    if (tr) {
      node = rc;
      continue;
    }
    if (top > bottom) {
      node = start = stack[--top & (kStack - 1)];
      continue;
    }
    if (bottom == 0) return;  // nothing was dropped
    // climb from the finished subtree to the next right child that was dropped
    for (node = start; moves > 0; --moves) {
      if (node == root) return;
      const int up = __ldg(parent + node), r = __ldg(right + up);
      if (node != r && r >= n && accept(r)) {
        node = start = r;
        break;
      }
      node = up;
    }
  }
}

}  // namespace ar_lbvh
