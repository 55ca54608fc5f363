// The reference's sequential-impulse path (updateUniformGridSIS, RigidBodies/UniformGridUpdate.cpp
// :734-815) on the GPU, in REFERENCE semantics: per-particle deepest contact on the uniform grid,
// the contact list in particle order, and the Gauss-Seidel impulse iterations.  The reference
// runs the last two on the host (Particles/updateFunctions.cpp:1431-1874) with a device round
// trip every step.
//
// The solver is exact, not a parallel approximation.  A contact's update reads and writes only
// the velocities of its (one or two) bodies and its own accumulated impulses, so two contacts
// that share no body commute.  Contacts are therefore given levels -- level(c) = 1 + the highest
// level among earlier contacts on either of its bodies -- and one level at a time is solved in
// parallel: every body sees exactly the sequence of updates of the reference's loop, so the
// results are the reference's bit for bit.  The level assignment is the same in every
// iteration, since it depends only on which bodies each contact touches, and the iterations
// are laid onto one schedule in which each starts before the previous one ends (see the
// schedule notes above sis_levels_kernel).
#include <algorithm>
#include <climits>

#include "ar_glm.cuh"
#include "ar_grid.cuh"
#include "ar_internal.cuh"

namespace {

using ar_glm::cross3;
using ar_glm::dot3;
using ar_glm::mv;

__device__ __forceinline__ float3 f3(float4 a) { return ar::mk3(a.x, a.y, a.z); }
__device__ __forceinline__ float3 add3(float3 a, float3 b) { return ar::add(a, b); }
__device__ __forceinline__ float3 sub3(float3 a, float3 b) { return ar::sub(a, b); }
__device__ __forceinline__ float3 mul3(float s, float3 a) { return ar::mk3(s * a.x, s * a.y, s * a.z); }
// x / y for the solver's updates.  A zero dividend over a finite non-zero divisor gives the
// signed zero that IEEE division gives (sign = sign of x xor sign of y) without dividing;
// bodies at rest make such quotients common, and the shortcut keeps them off the dependent
// chain of the update.  Every other case is the division itself.
__device__ __forceinline__ float qdiv(float x, float y) {
  if (x == 0.f && isfinite(y) && y != 0.f) return signbit(y) ? -x : x;
  return x / y;
}
__device__ __forceinline__ float3 qdiv3(float3 a, float s) {
  return ar::mk3(qdiv(a.x, s), qdiv(a.y, s), qdiv(a.z, s));
}
// glm::normalize(vec3): v * inversesqrt(dot(v, v)), inversesqrt(x) = 1 / sqrt(x)
__device__ __forceinline__ float3 gnormalize(float3 v) {
  const float inv = 1.0f / sqrtf(dot3(v, v));
  return ar::mk3(v.x * inv, v.y * inv, v.z * inv);
}

// ---- FindRigidBodyCollisionsUniformGridKernel (Kernels/RB_UniformGridKernels.cu:731-842) --------
// Per sorted particle: over the 27 neighbour cells (z, y, x = -1..1), occupants of other bodies;
// the deepest penetration 2r - |p - q| above the running maximum is kept with the other particle's
// original index and body.
__global__ void __launch_bounds__(128) find_contacts_grid_kernel(
    ar_grid::Grid g, float radius, const int32_t* __restrict__ rb_idx,
    const float4* __restrict__ spos, const uint32_t* __restrict__ gidx,
    const uint32_t* __restrict__ cstart, const uint32_t* __restrict__ cend, int n,
    float* __restrict__ contact_distance, int32_t* __restrict__ colliding_body,
    int32_t* __restrict__ colliding_particle) {
  const int index = blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= n) return;
  const float3 pos = f3(__ldg(spos + index));
  const int3 gp = g.cell_of(pos);
  const uint32_t orig = __ldg(gidx + index);
  const int body = __ldg(rb_idx + orig);
  const float threshold = 2 * radius;
  const float reach2_up = nextafterf(threshold * threshold, INFINITY);
  float best = contact_distance[orig];
  int best_particle = -1, best_body = 0;
  ar_grid::for_occupied(g, gp, cstart, cend, [&](uint32_t st, uint32_t en) {
    for (uint32_t j = st; j < en; ++j) {
      const float3 d = sub3(pos, f3(__ldg(spos + j)));
      const float d2 = ar::dot(d, d);
      // from the square just above threshold^2 on, the root is at least the threshold
      if (best >= 0.f && !(d2 < reach2_up)) continue;
      const float depth = threshold - sqrtf(d2);
      if (!(depth > best) || j == (uint32_t)index) continue;
      const int o2 = (int)__ldg(gidx + j);
      const int b2 = __ldg(rb_idx + o2);
      if (b2 == body) continue;
      best = depth;
      best_particle = o2;
      best_body = b2;
    }
  });
  if (best_particle >= 0) {
    contact_distance[orig] = best;
    colliding_particle[orig] = best_particle;
    colliding_body[orig] = best_body;
  }
}

// ---- GatherRigidBodyCollisions (Particles/updateFunctions.cpp:1431-1500) -----------------------
// Particles with a contact (distance > 0), in particle order, become contacts: the contact point
// and normal of findExactContactPoint (Particles/CPU_Engine.cpp:461-473, float4 arithmetic with
// helper_math's host normalize, 1 / sqrt), the bias restitution * relative normal velocity, and
// zeroed accumulated impulses.  Order-preserving compaction: per-block counts, their scan, and
// the scatter.
constexpr int kGatherBlock = 256;

__global__ void __launch_bounds__(kGatherBlock) gather_count_kernel(
    const float* __restrict__ contact_distance, int n, int* __restrict__ block_counts) {
  const int i = blockIdx.x * kGatherBlock + threadIdx.x;
  const bool hit = i < n && __ldg(contact_distance + i) > 0.f;
  const int c = __syncthreads_count(hit);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = c;
}

// Exclusive scan of the block counts in one block (any number of blocks, 1024 at a time).
__global__ void __launch_bounds__(1024) gather_scan_kernel(int* __restrict__ block_counts,
                                                           int blocks, int* __restrict__ total) {
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < blocks; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < blocks ? block_counts[i] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    const int carry = s_carry;
    const int excl = carry + (warp > 0 ? s_warp[warp - 1] : 0) + x - v;
    if (i < blocks) block_counts[i] = excl;
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = s_carry;
}

__global__ void __launch_bounds__(kGatherBlock) gather_write_kernel(
    float radius, float restitution, const int32_t* __restrict__ rb_idx,
    const float4* __restrict__ cms, const float4* __restrict__ vel, const float4* __restrict__ ang,
    const float4* __restrict__ rel, const float* __restrict__ contact_distance,
    const int32_t* __restrict__ colliding_body, const int32_t* __restrict__ colliding_particle,
    int n, const int* __restrict__ block_offsets, int capacity, float4* __restrict__ normal,
    float4* __restrict__ point, int32_t* __restrict__ body1, int32_t* __restrict__ body2,
    float* __restrict__ bias, float* __restrict__ acc_impulse, float* __restrict__ acc_friction,
    float* __restrict__ acc_friction2, int* __restrict__ err) {
  __shared__ int s_warp[kGatherBlock / 32];
  const int i = blockIdx.x * kGatherBlock + threadIdx.x;
  const bool hit = i < n && __ldg(contact_distance + i) > 0.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t m = __ballot_sync(0xffffffffu, hit);
  if (lane == 0) s_warp[warp] = __popc(m);
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (!hit) return;
  const int c = block_offsets[blockIdx.x] + before + __popc(m & ((1u << lane) - 1));
  if (c >= capacity) {
    ar::raise_error(err, ar::kErrOverflow);
    return;
  }
  const int b = __ldg(rb_idx + i);
  const int j = __ldg(colliding_particle + i);
  const int b2 = __ldg(colliding_body + i);
  const float4 cm1 = __ldg(cms + b), cm2 = __ldg(cms + b2);
  const float4 r1 = __ldg(rel + i), r2 = __ldg(rel + j);
  const float4 p1 = make_float4(cm1.x + r1.x, cm1.y + r1.y, cm1.z + r1.z, cm1.w + r1.w);
  const float4 p2 = make_float4(cm2.x + r2.x, cm2.y + r2.y, cm2.z + r2.z, cm2.w + r2.w);
  const float t = radius / (radius + radius);
  const float4 cp = make_float4(p1.x + (p2.x - p1.x) * t, p1.y + (p2.y - p1.y) * t,
                                p1.z + (p2.z - p1.z) * t, p1.w + (p2.w - p1.w) * t);
  const float4 d = make_float4(p2.x - p1.x, p2.y - p1.y, p2.z - p1.z, p2.w - p1.w);
  const float inv = 1.0f / sqrtf(d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w);
  const float4 cn = make_float4(d.x * inv * (-1.f), d.y * inv * (-1.f), d.z * inv * (-1.f),
                                d.w * inv * (-1.f));
  const float3 n3 = f3(cn);
  const float3 v1 = f3(__ldg(vel + b)), w1 = f3(__ldg(ang + b));
  const float3 v2 = f3(__ldg(vel + b2)), w2 = f3(__ldg(ang + b2));
  const float v_rel = ar::dot(add3(v1, ar::cross(w1, f3(r1))), n3) -
                      ar::dot(add3(v2, ar::cross(w2, f3(r2))), n3);
  normal[c] = cn;
  point[c] = cp;
  body1[c] = b;
  body2[c] = b2;
  bias[c] = restitution * v_rel;
  acc_impulse[c] = 0.f;
  acc_friction[c] = 0.f;
  acc_friction2[c] = 0.f;
}

// ---- SequentialImpulseSolver (Particles/updateFunctions.cpp:1580-1874) --------------------------
struct Contacts {
  const float4* normal;
  const float4* point;
  const int32_t* body1;
  const int32_t* body2;
  const float* bias;
  float* acc_impulse;
  float* acc_friction;
  float* acc_friction2;
};
struct Bodies {
  const float4* cms;
  float4* vel;
  float4* ang;
  const float* inv_inertia;  // current (world) inverse inertia, glm::mat3
  const float* mass;
};

__device__ __forceinline__ float clampf(float v, float lo, float hi) {
  return v < lo ? lo : (v > hi ? hi : v);
}

// One contact's update, the reference's loop body.  The reference compares the float values
// with double constants (abs(x) < 0.00001), so the comparisons are made in double here too.
// A contact's geometry: everything in its update that does not depend on the velocities --
// the lever arms, the effective mass mc (set to 1 below 1e-5, as the reference does), the two
// tangent directions and their effective masses, and the friction bound.  It is the same in
// every sweep, so it is computed once, with the reference's expressions, before the sweeps.
struct Geometry {
  float4 g0;  // p1, mc
  float4 g1;  // p2, friction bound
  float4 g2;  // t1, k1
  float4 g3;  // t2, k2
};

__device__ Geometry contact_geometry(float3 n, float4 point, float4 cm1, float4 cm2,
                                     const float* I1, const float* I2, float m1, float m2,
                                     bool two_body, float ar_friction, float rb_friction,
                                     float abs_gravity_y) {
  const float3 p1 = ar::mk3(point.x - cm1.x, point.y - cm1.y, point.z - cm1.z);
  float3 p2 = ar::mk3(0.f, 0.f, 0.f);
  float mc, bound, k1, k2;
  float3 t1 = ar::mk3(1.f, 0.f, 0.f);
  if (!two_body) {
    mc = 1 / m1 + dot3(cross3(mv(I1, cross3(p1, n)), p1), n);
    if ((double)fabsf(mc) < 0.00001) mc = 1.f;
    bound = ar_friction * mc * abs_gravity_y;
    if ((double)fabsf(t1.x - n.x) < 0.0001) t1 = ar::mk3(0.f, 1.f, 0.f);
    else if ((double)fabsf(t1.x + n.x) < 0.0001) t1 = ar::mk3(0.f, 1.f, 0.f);
    t1 = gnormalize(sub3(t1, mul3(dot3(t1, n), n)));
    k1 = 1 / m1 + dot3(cross3(mv(I1, cross3(p1, t1)), p1), t1);
  } else {
    p2 = ar::mk3(point.x - cm2.x, point.y - cm2.y, point.z - cm2.z);
    mc = 1 / m1 + 1 / m2 + dot3(cross3(mv(I1, cross3(p1, n)), p1), n) +
         dot3(cross3(mv(I2, cross3(p2, n)), p2), n);
    if ((double)fabsf(mc) < 0.00001) mc = 1.f;
    bound = rb_friction * mc * abs_gravity_y;
    if ((double)fabsf(t1.x - n.x) < 0.0001) t1 = ar::mk3(0.f, 1.f, 0.f);
    t1 = gnormalize(sub3(t1, mul3(dot3(t1, n), n)));
    k1 = (1 / m1 + dot3(cross3(mv(I1, cross3(p1, t1)), p1), t1)) +
         (1 / m2 + dot3(cross3(mv(I2, cross3(p2, t1)), p2), t1));
  }
  const float3 t2 = gnormalize(cross3(t1, n));
  if (!two_body)
    k2 = 1 / m1 + dot3(cross3(mv(I1, cross3(p1, t2)), p1), t2);
  else
    k2 = (1 / m1 + dot3(cross3(mv(I1, cross3(p1, t2)), p1), t2)) +
         (1 / m2 + dot3(cross3(mv(I2, cross3(p2, t2)), p2), t2));
  return Geometry{make_float4(p1.x, p1.y, p1.z, mc), make_float4(p2.x, p2.y, p2.z, bound),
                  make_float4(t1.x, t1.y, t1.z, k1), make_float4(t2.x, t2.y, t2.z, k2)};
}

// Geometry of every contact (one thread per contact).
__global__ void __launch_bounds__(256) sis_geometry_kernel(
    Contacts C, Bodies B, const int* __restrict__ d_count, int capacity, float ar_friction,
    float rb_friction, float abs_gravity_y, Geometry* __restrict__ geo) {
  const int count = min(*d_count, capacity);
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < count; c += gridDim.x * blockDim.x) {
    const int i1 = C.body1[c], i2 = C.body2[c];
    const bool two = i2 >= 0;
    geo[c] = contact_geometry(f3(C.normal[c]), C.point[c], B.cms[i1],
                              two ? B.cms[i2] : make_float4(0.f, 0.f, 0.f, 0.f),
                              B.inv_inertia + 9 * i1, B.inv_inertia + 9 * (two ? i2 : i1),
                              B.mass[i1], two ? B.mass[i2] : 1.f, two, ar_friction, rb_friction,
                              abs_gravity_y);
  }
}

// x / d for the solver's divisors, which do not change from sweep to sweep, from r = 1 / d: two
// residual corrections of x * r.  The first leaves an error well below one unit in the last place,
// and then the second one's result is the correctly rounded quotient, since r is the correctly
// rounded reciprocal and the residual is exact (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990).  Holds for |x| and d in the ranges tested below, in
// which nothing over- or underflows; a zero dividend gives the zero of IEEE division's sign.
__device__ __forceinline__ float div_by(float x, float d, float r) {
  const float q0 = x * r;
  const float q1 = fmaf(fmaf(-q0, d, x), r, q0);
  const float q2 = fmaf(fmaf(-q1, d, x), r, q1);
  return copysignf(q2, q0);
}
__device__ __forceinline__ bool div_dividend(float x) {  // zero, or 2^-70 <= |x| < 2^60
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u - 0x1c800000u < 0x5d800000u - 0x1c800000u || u == 0;
}
__device__ __forceinline__ bool div_divisor(float d) {  // 2^-40 <= |d| < 2^40
  const uint32_t u = __float_as_uint(d) & 0x7fffffffu;
  return u - 0x2b800000u < 0x53800000u - 0x2b800000u;
}

// A contact in the solver's working order: two halves, one per body, solved by two neighbouring
// lanes.  A half is five float4 words, stored in blocks of 32 halves, word by word, so that a warp
// loading consecutive contacts reads each word as one or two contiguous runs (half h of the packed
// order at half_at(h), its words 32 apart; the halves of contact p are 2 p and 2 p + 1):
//   normal, bias | lever arm, mc | inverse inertia 0..3 | 4..7 |
//   inverse inertia 8, mass, 1 / mass, body and flags
// The second half's inverse inertia, mass and 1 / mass are negated: its body takes the opposite
// impulse, and negated factors give exactly the negated products, sums and quotients.
// A contact with one body has no second half; its place holds what the first one's friction needs:
//   t1, k1 | t2, k2 | 1 / mc, 1 / k1, 1 / k2, - | - | friction bound, 0, 0, kNoBody
// Beside them two floats per half that change: the impulse and the number of sweeps done (first
// half); 1 / mc, or a one-body contact's two frictions (second half).
// kOdd marks the contacts that the plain form of solve_half does not cover: those with one body,
// with one body twice, or with a divisor outside div_by's range, whose reciprocal is a NaN here.
constexpr int kHalfWords = 5;
constexpr uint32_t kOdd = 1u << 31, kNoBody = 0xffffffffu;
__device__ __forceinline__ float reciprocal(float d) {
  return div_divisor(d) ? 1.0f / d : __int_as_float(0x7fc00000);
}
__device__ __forceinline__ size_t half_at(int h) {
  return (size_t)(h >> 5) * (32 * kHalfWords) + (h & 31);
}
// Returns whether the contact is odd.
__device__ __forceinline__ bool pack_contact(const Contacts& C, const Bodies& B,
                                             const Geometry* __restrict__ geo, int c, int p,
                                             float4* __restrict__ rec,
                                             float2* __restrict__ accs) {
  const int i1 = C.body1[c], i2 = C.body2[c];
  const float4 n = C.normal[c];
  const Geometry g = geo[c];
  const float mc = g.g0.w, m1 = B.mass[i1], m2 = i2 >= 0 ? B.mass[i2] : m1;
  const bool odd = i2 < 0 || i2 == i1 || !div_divisor(mc) || !div_divisor(m1) || !div_divisor(m2);
  auto half = [&](int side, float4 arm, int body, float mass) {
    const float sign = side ? -1.f : 1.f, m = sign * mass;
    float I[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) I[k] = sign * B.inv_inertia[9 * (size_t)body + k];
    float4* out = rec + half_at(2 * p + side);
    out[0] = make_float4(n.x, n.y, n.z, C.bias[c]);
    out[32] = make_float4(arm.x, arm.y, arm.z, mc);
    out[64] = make_float4(I[0], I[1], I[2], I[3]);
    out[96] = make_float4(I[4], I[5], I[6], I[7]);
    out[128] = make_float4(I[8], m, reciprocal(m),
                           __uint_as_float((uint32_t)body | (odd ? kOdd : 0u)));
  };
  half(0, g.g0, i1, m1);
  if (i2 >= 0) {
    half(1, g.g1, i2, m2);
  } else {
    float4* out = rec + half_at(2 * p + 1);
    out[0] = g.g2;
    out[32] = g.g3;
    out[64] = make_float4(reciprocal(mc), reciprocal(g.g2.w), reciprocal(g.g3.w), 0.f);
    out[128] = make_float4(g.g1.w, 0.f, 0.f, __uint_as_float(kNoBody));
  }
  accs[2 * (size_t)p] = make_float2(C.acc_impulse[c], __int_as_float(0));
  accs[2 * (size_t)p + 1] = i2 >= 0 ? make_float2(reciprocal(mc), 0.f)
                                    : make_float2(C.acc_friction[c], C.acc_friction2[c]);
  return odd;
}

// Half of a contact, held in registers (h: its place, -1: none).
struct Half {
  float4 w[kHalfWords];
  float2 acc;
  int h;
};
// Loads at this point of the program: the compiler would move plain loads down to their uses, a
// step later, to save registers.  Through L1, which holds a small list: its steps are shorter than
// two steps' way to L2 (200 bodies in a chain, 300 sweeps: 1.24 -> 1.14 ms, 27 cubes of 8 0.75 ->
// 0.63; large lists the same).
__device__ __forceinline__ float4 load_now(const float4* p) {
  float4 v;
  asm volatile("ld.global.ca.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float2 load_now(const float2* p) {
  float2 v;
  asm volatile("ld.global.ca.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void load_half(const float4* rec, const float2* accs, int h, Half& it) {
  it.h = h;
  if (h < 0) return;
  const float4* at = rec + half_at(h);
#pragma unroll
  for (int k = 0; k < kHalfWords; ++k) it.w[k] = load_now(at + 32 * k);
  it.acc = load_now(accs + h);
}

// What an update leaves to be stored: no other update waits for it, so it is done in the next
// step, between that step's dependent operations.
struct Rest {
  int h = -1, sweep;
  float total;
  float3 v, c;  // the body's velocity before the update, and angular velocity x lever arm
  bool slides = false;  // between two bodies
};
// The accumulated impulse, and the relative velocity for the friction as the reference sums it.
template <bool kGeneral>
__device__ __forceinline__ void store_rest(const Rest& r, float2* __restrict__ accs,
                                           float4* __restrict__ vrel, size_t stride) {
  const bool first = r.h >= 0 && !(threadIdx.x & 1);
  if (first) accs[r.h] = make_float2(r.total, __int_as_float(r.sweep + 1));
  if (kGeneral && !__any_sync(0xffffffffu, r.slides)) return;
  auto pair = [&](float x) { return __shfl_xor_sync(0xffffffffu, x, 1); };
  const float3 v2 = ar::mk3(pair(r.v.x), pair(r.v.y), pair(r.v.z));
  const float3 c2 = ar::mk3(pair(r.c.x), pair(r.c.y), pair(r.c.z));
  const float3 slide = add3(add3(add3(mul3(-1.f, r.v), r.c), v2), c2);
  if (first && (!kGeneral || r.slides))
    vrel[(size_t)r.sweep * stride + (r.h >> 1)] = make_float4(slide.x, slide.y, slide.z, 0.f);
}
// One contact's update, the velocity-dependent part of the reference's loop body, by the two
// lanes that hold its halves (every lane of the warp calls it).  Each lane takes its body's share
// of the relative velocity, both compute the impulse, and each updates its body.  Friction between
// two bodies is accumulated but never applied (as in the reference), so only the relative velocity
// it needs is kept, in `vrel`, for sis_friction_kernel.  Lanes without a contact compute along on
// what their registers hold, so they must not decide on a warp's plain division.  kGeneral: some
// contact of the list is odd (else the compiler leaves the tests for it out).
template <bool kGeneral>
__device__ __forceinline__ void solve_half(const Half& it, float2* __restrict__ accs, float4* vel,
                                           float4* ang, float4* __restrict__ vrel, size_t stride,
                                           float upper_bound, Rest& rest) {
  constexpr uint32_t kAll = 0xffffffffu;
  const bool side = threadIdx.x & 1;
  const bool have = it.h >= 0;
  const uint32_t tag = have ? __float_as_uint(it.w[4].w) : 0u;
  const bool mine = have && tag != kNoBody;  // this lane holds a body
  const int body = mine ? (int)(tag & ~kOdd) : 0;
  const float3 n = f3(it.w[0]), arm = f3(it.w[1]);
  const float mc = it.w[1].w, m = it.w[4].y;
  const float3 v = f3(vel[body]), w = f3(ang[body]);
  // of a general list, the warps with an odd contact (the whole warp takes a branch on `some`)
  const bool odd = kGeneral && (tag & kOdd);
  const bool some = kGeneral && __any_sync(kAll, odd);
  const uint32_t other = some ? __shfl_xor_sync(kAll, tag, 1) : tag;
  const bool one = odd && (side ? tag : other) == kNoBody;
  store_rest<kGeneral>(rest, accs, vrel, stride);  // the previous update's
  // the first lane's impulse against the second one's 1 / mc
  const float met = __shfl_xor_sync(kAll, it.acc.x, 1);
  const float acc = side ? met : it.acc.x;
  float rmc = side ? it.acc.x : met;
  if (some) {
    const float r = __shfl_xor_sync(kAll, it.w[2].x, 1);
    if (one) rmc = r;
  }
  const float3 c = cross3(w, arm);
  const float3 at = add3(v, c);  // the body's velocity at the contact
  const float s = dot3(at, n);
  const float d = s - __shfl_xor_sync(kAll, s, 1);
  const float v_rel = one ? s : (side ? -d : d);
  const float x = -(v_rel + it.w[0].w);
  float change = div_by(x, mc, rmc);
  if (mine && !(div_dividend(x) && (!kGeneral || rmc == rmc))) change = x / mc;
  const float total = clampf(acc + change, 0.f, upper_bound);
  float3 imp = mul3(total - acc, n);
  if (some) {
    // one body: the second lane computes the frictions, which are applied
    auto pair = [&](float3 a) {  // the other half's
      return ar::mk3(__shfl_xor_sync(kAll, a.x, 1), __shfl_xor_sync(kAll, a.y, 1),
                     __shfl_xor_sync(kAll, a.z, 1));
    };
    const float3 vel1 = pair(at);
    const bool friction = one && side;
    const float x1 = -dot3(vel1, n), x2 = -dot3(vel1, arm);  // along t1 and t2
    float cf1 = div_by(x1, it.w[0].w, it.w[2].y), cf2 = div_by(x2, mc, it.w[2].z);
    if (friction && !(div_dividend(x1) && div_dividend(x2) && it.w[2].y == it.w[2].y &&
                      it.w[2].z == it.w[2].z)) {
      cf1 = x1 / it.w[0].w;
      cf2 = x2 / mc;
    }
    const float bound = it.w[4].x;
    const float f1 = clampf(it.acc.x + cf1, -bound, bound);
    cf1 = f1 - it.acc.x;
    const float f2 = clampf(it.acc.y + cf2, -bound, bound);
    cf2 = f2 - it.acc.y;
    if (friction) accs[it.h] = make_float2(f1, f2);
    const float3 fx = pair(mul3(cf1, n)), fy = pair(mul3(cf2, arm));
    if (one) imp = add3(add3(imp, fx), fy);
  }
  const float rm = it.w[4].z;
  float3 dv = ar::mk3(div_by(imp.x, m, rm), div_by(imp.y, m, rm), div_by(imp.z, m, rm));
  if (mine && !(div_dividend(imp.x) && div_dividend(imp.y) && div_dividend(imp.z) &&
                (!kGeneral || rm == rm)))
    dv = ar::mk3(imp.x / m, imp.y / m, imp.z / m);
  const float I[9] = {it.w[2].x, it.w[2].y, it.w[2].z, it.w[2].w, it.w[3].x,
                      it.w[3].y, it.w[3].z, it.w[3].w, it.w[4].x};
  const float3 nv = add3(v, dv), nw = add3(w, mv(I, cross3(arm, imp)));
  // of a contact of one body with itself the second half's update stands
  if (mine && (side || !odd || tag != other)) {
    vel[body] = make_float4(nv.x, nv.y, nv.z, 0.f);
    ang[body] = make_float4(nw.x, nw.y, nw.z, 0.f);
  }
  rest = Rest{it.h, __float_as_int(it.acc.y), total, v, c, have && !one};
}

// Threads of the sweep block, two lanes per contact: a step's first 320 contacts are loaded ahead.
// The block keeps as many warps as its widest step fills; idle ones would cost every step a little.
constexpr int kSisThreads = 640;
constexpr int kLevelChunk = 1024;  // body pairs staged per step of the level walk
constexpr int kLayoutThreads = 1024;
constexpr size_t kSisSmemMax = 220 * 1024;   // the sweep block's dynamic shared memory
constexpr size_t kWalkSmemMax = 200 * 1024;  // the walk's (its static 16 KB stay below 227 KB)
// Relative velocities kept at most, 16 bytes each (one per contact and sweep of a schedule).
constexpr long long kMaxSlots = 1l << 25;
// The schedule's header in scratch memory: levels, shift, contact count, whether some contact is odd,
// and sweeps per schedule.
enum {
  kHdrLevels = 0, kHdrShift = 1, kHdrCount = 2, kHdrGeneral = 3, kHdrSweeps = 4, kHdrWords = 8
};

// Schedule.  Each contact gets a level: 1 + the highest level among earlier contacts on either
// of its bodies.  Sweep s solves level b at step b + s * shift of one schedule, where shift
// exceeds the span of levels that any body's contacts cover.  Then no step holds two contacts
// of one body (two items of one step from sweeps s < s' on body x would need levels of x at
// least shift apart), and each body's updates come in the reference's order: within a sweep
// by level, and the last of sweep s (at step <= first + span + s * shift) before the first of
// sweep s + 1.  Every update therefore reads exactly the values the reference's loop gives it,
// while consecutive sweeps overlap.  Step l covers the levels b congruent to l (mod shift)
// with max(1, l - (iterations - 1) shift) <= b <= min(levels, l), so the contacts are packed
// by (level mod shift, level) and each step's contacts are one contiguous run.

// Levels, each body's first and last level, the span and the shift.  The block stages the
// contacts' body pairs in shared memory, the next chunk while warp 0 walks this one in order, a
// run at a time: a run is up to 32 consecutive contacts on one first body A (the gather emits each
// body's contacts together).  Inside a run, with x_j the last level of contact j's other body
// before the run, level_j = 1 + max(level_{j-1}, x_j): A's last level is the previous
// contact's, and an other body met earlier in the same run was last touched at a level no
// higher than level_{j-1}.  Unrolled, level_j = j + 1 + max(last level of A, max_{i<=j}
// (x_i - i)), a prefix maximum over the warp's lanes.  A body's last level is then the level
// of its last contact in the run (atomicMax), its first level the level of its first contact
// when it had none before (atomicMin).  Any order of contacts is walked correctly; short runs
// only leave lanes idle.
// Bound by one warp's chain from run to run, so the chain is kept short: the next run's pairs are
// read during this one, the prefix maximum stops at the run's length, and A's last level is stored
// by the lane that has it (4,096 packed cubes: 1450 -> 986 us).
// kShared: the walk's last / first levels live in shared memory.
template <bool kShared>
__global__ void __launch_bounds__(256) sis_levels_kernel(
    const int32_t* __restrict__ body1, const int32_t* __restrict__ body2,
    const int* __restrict__ d_count, int capacity, int num_bodies, int* __restrict__ level,
    int* __restrict__ last, int* __restrict__ first, int iterations, long long slots,
    int* __restrict__ hdr, int* __restrict__ err) {
  extern __shared__ int s_walk[];
  __shared__ int2 s_pair[2][kLevelChunk];
  __shared__ int s_span, s_top;
  int count = *d_count;
  if (count > capacity) {
    if (threadIdx.x == 0) ar::raise_error(err, ar::kErrOverflow);
    count = capacity;
  }
  int* lastp = kShared ? s_walk : last;
  int* firstp = kShared ? s_walk + num_bodies : first;
  for (int b = threadIdx.x; b < num_bodies; b += blockDim.x) {
    lastp[b] = 0;
    firstp[b] = INT_MAX;
  }
  if (threadIdx.x == 0) s_span = s_top = 0;
  const int lane = threadIdx.x & 31;
  int top = 0;
  for (int i = threadIdx.x; i < min(kLevelChunk, count); i += blockDim.x)
    s_pair[0][i] = make_int2(body1[i], body2[i]);
  __syncthreads();
  for (int base = 0, buf = 0; base < count; base += kLevelChunk, buf ^= 1) {
    const int m = min(kLevelChunk, count - base);
    if (threadIdx.x >= 32) {  // the next chunk
      const int from = base + kLevelChunk, mn = min(kLevelChunk, count - from);
      for (int i = threadIdx.x - 32; i < mn; i += blockDim.x - 32)
        s_pair[buf ^ 1][i] = make_int2(body1[from + i], body2[from + i]);
    } else {
      const int2* pairs = s_pair[buf];
      const int2 none = make_int2(-1, -1);
      int2 pr = lane < m ? pairs[lane] : none;
      int a = pairs[0].x;
      for (int i = 0; i < m;) {  // one run (cut at 32 contacts and at the chunk's end)
        const uint32_t off = ~__ballot_sync(0xffffffffu, pr.x == a);
        const int k = off ? __ffs(off) - 1 : 32;  // contacts in the run (lane 0 is one)
        const bool in = lane < k;
        const int b = in && pr.y >= 0 && pr.y != a ? pr.y : -1;  // a self pair touches A only
        const int x = b >= 0 ? lastp[b] : 0;
        const int a_last = lastp[a];
        // the next run's pairs are on their way during this one
        const int next = i + k;
        const int2 pr_next = next + lane < m ? pairs[next + lane] : none;
        const int a_next = next < m ? pairs[next].x : 0;
        int y = in ? x - lane : INT_MIN / 2;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          if (d >= k) break;
          const int t = __shfl_up_sync(0xffffffffu, y, d);
          if (lane >= d) y = max(y, t);
        }
        const int l = lane + 1 + max(a_last, y);
        if (b >= 0) {
          atomicMax(lastp + b, l);
          if (x == 0) atomicMin(firstp + b, l);
        }
        if (lane == k - 1) lastp[a] = l;
        if (lane == 0 && a_last == 0) firstp[a] = l;
        if (in) {
          level[base + i + lane] = l;
          top = max(top, l);
        }
        i = next;
        pr = pr_next;
        a = a_next;
        __syncwarp();
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) atomicMax(&s_top, top);
  int span = 0;
  for (int b = threadIdx.x; b < num_bodies; b += blockDim.x)
    if (firstp[b] != INT_MAX) span = max(span, lastp[b] - firstp[b]);
  atomicMax(&s_span, span);
  __syncthreads();
  if (threadIdx.x == 0) {
    hdr[kHdrLevels] = s_top;
    hdr[kHdrShift] = max(4, s_span + 1);
    hdr[kHdrCount] = count;
    hdr[kHdrGeneral] = 0;
    hdr[kHdrSweeps] = (int)min((long long)iterations, slots / max(count, 1));
  }
}

// Level sizes (run[l].y, zeroed before).
__global__ void __launch_bounds__(256) sis_sizes_kernel(const int* __restrict__ level,
                                                        const int* __restrict__ hdr,
                                                        int2* __restrict__ run) {
  const int count = hdr[kHdrCount];
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < count; c += gridDim.x * blockDim.x)
    atomicAdd(&run[level[c]].y, 1);
}

// Position of level l in (level mod shift, level) order: class 0 (shift, 2 shift, ...) first,
// then classes 1 .. shift - 1; with levels = Q shift + R, class r >= 1 holds Q + (r <= R)
// levels, so it starts at r Q + min(r - 1, R).
__device__ __forceinline__ int layout_index(int l, int shift, int q, int rem) {
  const int r = l % shift;
  return r == 0 ? l / shift - 1 : r * q + min(r - 1, rem) + (l - r) / shift;
}

// Lays the level runs out: tmp[layout_index(l)] = size of level l, an exclusive scan of tmp,
// then run[l] = (start, start).  tmp holds `levels` ints.
__global__ void __launch_bounds__(kLayoutThreads) sis_layout_kernel(const int* __restrict__ hdr,
                                                                    int2* __restrict__ run,
                                                                    int* __restrict__ tmp) {
  __shared__ int s_warp[kLayoutThreads / 32];
  __shared__ int s_carry;
  const int levels = hdr[kHdrLevels], shift = hdr[kHdrShift];
  const int q = levels / shift, rem = levels % shift;
  for (int l = 1 + threadIdx.x; l <= levels; l += blockDim.x)
    tmp[layout_index(l, shift, q, rem)] = run[l].y;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < levels; base += blockDim.x) {
    const int j = base + threadIdx.x;
    const int v = j < levels ? tmp[j] : 0;
    int x = v;  // inclusive warp scan
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += y;
      }
      s_warp[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const int carry = s_carry;
    const int excl = carry + (warp > 0 ? s_warp[warp - 1] : 0) + x - v;
    if (j < levels) tmp[j] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = excl + v;
    __syncthreads();
  }
  for (int l = 1 + threadIdx.x; l <= levels; l += blockDim.x) {
    const int start = tmp[layout_index(l, shift, q, rem)];
    run[l] = make_int2(start, start);
  }
}

// Each contact takes the next slot of its level's run (the order inside a level is free: its
// contacts share no body) and is packed there with its accumulators; order[p] = contact.
// Afterwards level l occupies [run[l].y, run[l].x).
__global__ void __launch_bounds__(256) sis_pack_kernel(Contacts C, Bodies B,
                                                       const Geometry* __restrict__ geo,
                                                       const int* __restrict__ level,
                                                       int* __restrict__ hdr,
                                                       int2* __restrict__ run,
                                                       int* __restrict__ order,
                                                       float4* __restrict__ rec,
                                                       float2* __restrict__ accs) {
  const int count = hdr[kHdrCount];
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < count; c += gridDim.x * blockDim.x) {
    const int p = atomicAdd(&run[level[c]].x, 1);
    order[p] = c;
    if (pack_contact(C, B, geo, c, p, rec, accs)) hdr[kHdrGeneral] = 1;
  }
}

// The sweeps of the schedule numbered `schedule`, out of `iterations`.
__device__ __forceinline__ int sweeps_of(int schedule, int iterations, const int* hdr) {
  const long long left = iterations - (long long)schedule * hdr[kHdrSweeps];
  return (int)max(0ll, min(left, (long long)hdr[kHdrSweeps]));
}

// After a schedule: the accumulated impulses back to the caller's arrays, and the frictions of the
// contacts between two bodies, sweep by sweep from the relative velocities that the sweeps kept
// (the reference accumulates them in its loop; nothing else reads them).  The sweep counts start
// again at zero for the next schedule.
__global__ void __launch_bounds__(256) sis_friction_kernel(Contacts C,
                                                           const Geometry* __restrict__ geo,
                                                           const int* __restrict__ hdr,
                                                           const int* __restrict__ order,
                                                           const float4* __restrict__ vrel,
                                                           int schedule, int iterations,
                                                           float2* __restrict__ accs) {
  const int count = hdr[kHdrCount], sweeps = sweeps_of(schedule, iterations, hdr);
  if (sweeps == 0) return;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < count; p += gridDim.x * blockDim.x) {
    const int c = order[p];
    const float impulse = accs[2 * (size_t)p].x;
    C.acc_impulse[c] = impulse;
    accs[2 * (size_t)p] = make_float2(impulse, __int_as_float(0));
    if (C.body2[c] < 0) {
      const float2 f = accs[2 * (size_t)p + 1];
      C.acc_friction[c] = f.x;
      C.acc_friction2[c] = f.y;
      continue;
    }
    const float bound = geo[c].g1.w;
    const float4 t1 = geo[c].g2, t2 = geo[c].g3;
    float f1 = C.acc_friction[c], f2 = C.acc_friction2[c];
    for (int s = 0; s < sweeps; ++s) {
      const float3 v = f3(__ldcg(vrel + (size_t)s * count + p));
      f1 = clampf(f1 + qdiv(-dot3(v, f3(t1)), t1.w), -bound, bound);
      f2 = clampf(f2 + qdiv(-dot3(v, f3(t2)), t2.w), -bound, bound);
    }
    C.acc_friction[c] = f1;
    C.acc_friction2[c] = f2;
  }
}

// The contacts of one step of the schedule, [lo, hi): the levels b congruent to the step (mod
// shift) with max(1, step - (sweeps - 1) shift) <= b <= min(levels, step).
__device__ __forceinline__ int2 step_range(int step, int levels, int sweeps, int shift,
                                           const int2* runs) {
  if (step > levels + (sweeps - 1) * shift) return make_int2(0, 0);
  const int most = min(step, levels), least = max(1, step - (sweeps - 1) * shift);
  const int hi = most - (most - step % shift + shift) % shift;  // largest such level
  const int lo = least + (step - least) % shift;                // smallest
  return lo <= hi && hi >= 1 ? make_int2(runs[lo].y, runs[hi].x) : make_int2(0, 0);
}

// Barrier of the block's first `lanes` threads.
__device__ __forceinline__ void lanes_barrier(int lanes) {
  asm volatile("bar.sync 1, %0;" ::"r"(lanes) : "memory");
}

// The steps of a schedule of `sweeps` sweeps, in order, with a barrier between them.  Each lane
// loads its half of a contact two steps ahead (record and accumulators), into the
// registers of the one it has just solved: its accumulators were last written one step after the
// last update, shift >= 4 steps before they are needed, so their writer has passed a barrier since.
// `lanes`: of the block, those that take part, a multiple of 32.
template <bool kGeneral>
__device__ __forceinline__ void run_schedule(int lanes, int levels, int shift, int stride,
                                             int sweeps, float upper_bound, const int2* runs,
                                             const float4* rec, float2* accs, float4* vel,
                                             float4* ang, float4* vrel, int2* s_range) {
  const int steps = levels + (sweeps - 1) * shift;  // fits in int: checked by the host
  const int table = lanes - 2;                      // steps per table, even; two more looked up
  const int lane = threadIdx.x;  // this lane's half in a step's first round
  Rest rest;
  rest.v = rest.c = ar::mk3(0.f, 0.f, 0.f);
  auto fetch = [&](int2 r, Half& it) {
    load_half(rec, accs, 2 * r.x + lane < 2 * r.y ? 2 * r.x + lane : -1, it);
  };
  auto solve = [&](Half& it, int2 r, int2 ahead) {
    if (__any_sync(0xffffffffu, it.h >= 0 || rest.h >= 0)) {
      solve_half<kGeneral>(it, accs, vel, ang, vrel, stride, upper_bound, rest);
      for (int h0 = 2 * r.x + lanes; h0 < 2 * r.y; h0 += lanes) {
        // contacts beyond one per lane pair
        load_half(rec, accs, h0 + lane < 2 * r.y ? h0 + lane : -1, it);
        solve_half<kGeneral>(it, accs, vel, ang, vrel, stride, upper_bound, rest);
      }
    }
    fetch(ahead, it);
    lanes_barrier(lanes);
  };
  Half a, b;
  for (int base = 1; base <= steps; base += table) {
    s_range[threadIdx.x] = step_range(base + (int)threadIdx.x, levels, sweeps, shift, runs);
    lanes_barrier(lanes);
    if (base == 1) {
      fetch(s_range[0], a);
      fetch(s_range[1], b);
    }
    const int count = min(table, steps - base + 1);
    // two buffers in turn (a register move would wait for the loads in flight); `table` is even, so
    // every table starts with the same buffer
    for (int i = 0; i < count; i += 2) {
      solve(a, s_range[i], s_range[i + 2]);
      if (i + 1 >= count) break;
      solve(b, s_range[i + 1], s_range[i + 3]);
    }
  }
  store_rest<kGeneral>(rest, accs, vrel, stride);
}

// The sweeps, in one block.  kShared: the bodies' velocities and angular velocities live in shared
// memory.
// Bound by the serial chain of steps and by issue on one SM: 8,052 steps of up to 282 contacts on
// 4,096 packed cubes, 0.9 us each: a contact's dependent operations, a barrier and 160
// instructions per warp (40 % of the SM's issue slots).  13.7 -> 7.3 ms against a lane per contact
// with divisions (510 instructions), its friction and its accumulators before the barrier, and
// loads one step ahead that the step did not cover.  Tried: a cluster of two or four blocks, each
// with all velocities and storing into the others' (a cluster barrier per step costs 0.7 us: 13
// ms); copying the first words to shared memory two steps ahead with cp.async (fewer stalls, a
// quarter more instructions: 9.7 ms); three register buffers (spills: 28 ms).
template <bool kShared>
__global__ void __launch_bounds__(kSisThreads) sis_sweep_kernel(
    Bodies B, const int* __restrict__ hdr, int num_bodies, int schedule, int iterations,
    float upper_bound, const int2* __restrict__ run, const float4* __restrict__ rec,
    float2* __restrict__ accs, float4* __restrict__ vrel) {
  extern __shared__ float4 s_bodies[];  // (kShared) vel[num_bodies], ang[num_bodies]
  __shared__ int2 s_range[kSisThreads];
  __shared__ int s_widest;
  const int levels = hdr[kHdrLevels], shift = hdr[kHdrShift], count = hdr[kHdrCount];
  const int sweeps = sweeps_of(schedule, iterations, hdr);
  if (sweeps == 0 || levels == 0) return;
  float4 *vel = B.vel, *ang = B.ang;
  if (threadIdx.x == 0) s_widest = 0;
  if (kShared) {
    vel = s_bodies;
    ang = s_bodies + num_bodies;
    for (int b = threadIdx.x; b < num_bodies; b += blockDim.x) {
      vel[b] = B.vel[b];
      ang[b] = B.ang[b];
    }
  }
  __syncthreads();
  int widest = 0;
  const int steps = levels + (sweeps - 1) * shift;
  for (int step = 1 + (int)threadIdx.x; step <= steps; step += kSisThreads) {
    const int2 r = step_range(step, levels, sweeps, shift, run);
    widest = max(widest, r.y - r.x);
  }
  atomicMax(&s_widest, widest);
  __syncthreads();
  const int lanes = min((2 * s_widest + 31) & ~31, kSisThreads);
  if ((int)threadIdx.x >= lanes) return;
  if (hdr[kHdrGeneral])
    run_schedule<true>(lanes, levels, shift, count, sweeps, upper_bound, run, rec, accs, vel, ang,
                       vrel, s_range);
  else
    run_schedule<false>(lanes, levels, shift, count, sweeps, upper_bound, run, rec, accs, vel, ang,
                        vrel, s_range);
  if (kShared) {  // (each step ends with a barrier)
    for (int b = threadIdx.x; b < num_bodies; b += lanes) {
      B.vel[b] = vel[b];
      B.ang[b] = ang[b];
    }
  }
}

}  // namespace

extern "C" {

ar_status ar_find_contacts_grid(ar_ctx* ctx, const ar_sim_params* params, const int32_t* rb_idx,
                                const float* sorted_pos4, const uint32_t* grid_idx,
                                const uint32_t* cell_start, const uint32_t* cell_end, int n,
                                float* contact_distance, int32_t* colliding_body,
                                int32_t* colliding_particle, ar_stream_t stream) {
  if (!ctx || !params || n < 0 ||
      (n > 0 && (!rb_idx || !sorted_pos4 || !grid_idx || !cell_start || !cell_end ||
                 !contact_distance || !colliding_body || !colliding_particle)))
    return AR_ERR_INVALID_ARG;
  for (int a = 0; a < 3; ++a) {
    const uint32_t g = params->grid_size[a];
    if (!g || (g & (g - 1))) {
      arh::set_error("grid_size must be powers of two (the hash wraps with & (G-1))");
      return AR_ERR_INVALID_ARG;
    }
  }
  if (n == 0) return AR_OK;
  find_contacts_grid_kernel<<<arh::grid_for(n, 128), 128, 0, arh::stream(stream)>>>(
      ar_grid::Grid::from_params(*params), params->particle_radius, rb_idx,
      (const float4*)sorted_pos4, grid_idx, cell_start, cell_end, n, contact_distance,
      colliding_body, colliding_particle);
  return arh::check_launch("ar_find_contacts_grid");
}

ar_status ar_gather_contacts(ar_ctx* ctx, const ar_sim_params* params, int n,
                             const int32_t* rb_idx, const float* cms4, const float* vel4,
                             const float* ang4, const float* rel4, const float* contact_distance,
                             const int32_t* colliding_body, const int32_t* colliding_particle,
                             int capacity, float* normal4, float* point4, int32_t* body1,
                             int32_t* body2, float* bias, float* acc_impulse,
                             float* acc_friction, float* acc_friction2, int32_t* d_count,
                             ar_stream_t stream) {
  if (!ctx || !params || n < 0 || capacity < 0 || !d_count ||
      (n > 0 && (!rb_idx || !cms4 || !vel4 || !ang4 || !rel4 || !contact_distance ||
                 !colliding_body || !colliding_particle)) ||
      (capacity > 0 && (!normal4 || !point4 || !body1 || !body2 || !bias || !acc_impulse ||
                        !acc_friction || !acc_friction2)))
    return AR_ERR_INVALID_ARG;
  cudaStream_t st = arh::stream(stream);
  if (n == 0) {
    cudaMemsetAsync(d_count, 0, sizeof(int32_t), st);
    return arh::check_launch("ar_gather_contacts");
  }
  const int blocks = (int)arh::grid_for(n, kGatherBlock);
  int* offsets = (int*)arh::scratch(ctx, sizeof(int) * (size_t)blocks);
  if (!offsets) return AR_ERR_OOM;
  gather_count_kernel<<<blocks, kGatherBlock, 0, st>>>(contact_distance, n, offsets);
  gather_scan_kernel<<<1, 1024, 0, st>>>(offsets, blocks, d_count);
  gather_write_kernel<<<blocks, kGatherBlock, 0, st>>>(
      params->particle_radius, params->rb_restitution, rb_idx, (const float4*)cms4,
      (const float4*)vel4, (const float4*)ang4, (const float4*)rel4, contact_distance,
      colliding_body, colliding_particle, n, offsets, capacity, (float4*)normal4,
      (float4*)point4, body1, body2, bias, acc_impulse, acc_friction, acc_friction2, ctx->d_err);
  return arh::check_launch("ar_gather_contacts");
}

ar_status ar_sequential_impulse(ar_ctx* ctx, const ar_sim_params* params, const int32_t* d_count,
                                int capacity, const float* normal4, const float* point4,
                                const int32_t* body1, const int32_t* body2, const float* bias,
                                float* acc_impulse, float* acc_friction, float* acc_friction2,
                                int num_bodies, const float* cms4, float* vel4, float* ang4,
                                const float* cur_inv_inertia9, const float* mass, int iterations,
                                ar_stream_t stream) {
  if (!ctx || !params || !d_count || capacity < 0 || num_bodies < 0 || iterations < 0 ||
      (capacity > 0 && (!normal4 || !point4 || !body1 || !body2 || !bias || !acc_impulse ||
                        !acc_friction || !acc_friction2)) ||
      (num_bodies > 0 && (!cms4 || !vel4 || !ang4 || !cur_inv_inertia9 || !mass)))
    return AR_ERR_INVALID_ARG;
  if (capacity == 0 || num_bodies == 0 || iterations == 0) return AR_OK;
  // the schedule has at most capacity + (iterations - 1) (capacity + 1) steps, counted in int
  if ((long long)iterations * ((long long)capacity + 1) > INT_MAX) {
    arh::set_error("iterations x (capacity + 1) must stay below 2^31");
    return AR_ERR_INVALID_ARG;
  }
  // scratch: geometry[capacity] (64-byte aligned), the halves' records (word-major), the
  // accumulators, level runs run[capacity + 1], the schedule header, level[capacity],
  // order[capacity], last[num_bodies], first[num_bodies], then the relative velocities of a
  // schedule's sweeps.  These get room for all sweeps of `capacity` contacts, up to kMaxSlots, and
  // at least for one; the contacts that there are take what sweeps fit (kHdrSweeps), since the
  // results do not depend on where the sweeps are cut into schedules.
  const size_t cap = (size_t)capacity;
  const size_t geo_bytes = sizeof(Geometry) * cap;
  const size_t rec_bytes = sizeof(float4) * ((2 * cap + 31) / 32 * 32) * kHalfWords;
  const size_t acc_bytes = sizeof(float2) * 2 * cap;
  const size_t run_bytes = sizeof(int2) * (cap + 1);
  const size_t words = kHdrWords + 2 * cap + 2 * (size_t)num_bodies;
  const size_t fixed_bytes =
      (geo_bytes + rec_bytes + acc_bytes + run_bytes + sizeof(int) * words + 15) & ~(size_t)15;
  const long long want_slots =
      std::max((long long)capacity, std::min((long long)capacity * iterations, kMaxSlots));
  cudaStream_t st = arh::stream(stream);
  char* base = (char*)arh::scratch(ctx, fixed_bytes + sizeof(float4) * cap,
                                   fixed_bytes + sizeof(float4) * (size_t)want_slots, st);
  if (!base) return AR_ERR_OOM;
  const long long slots =
      std::min(want_slots, (long long)((ctx->scratch_bytes - fixed_bytes) / sizeof(float4)));
  Geometry* geo = (Geometry*)base;
  float4* rec = (float4*)(base + geo_bytes);
  float2* accs = (float2*)((char*)rec + rec_bytes);
  int2* run = (int2*)(accs + 2 * cap);
  int* hdr = (int*)(run + cap + 1);
  int* level = hdr + kHdrWords;
  int* order = level + capacity;
  int* last = order + capacity;
  int* first = last + num_bodies;
  float4* vrel = (float4*)(base + fixed_bytes);
  Contacts C{(const float4*)normal4, (const float4*)point4, body1, body2, bias, acc_impulse,
             acc_friction, acc_friction2};
  Bodies B{(const float4*)cms4, (float4*)vel4, (float4*)ang4, cur_inv_inertia9, mass};
  const unsigned gg = std::min(arh::grid_for(capacity, 256), (unsigned)ctx->num_sms * 8);
  sis_geometry_kernel<<<gg, 256, 0, st>>>(C, B, d_count, capacity, params->ar_friction,
                                          params->rb_friction, fabsf(params->gravity[1]), geo);
  cudaMemsetAsync(run, 0, run_bytes, st);
  // levels: the walk's last / first levels in shared memory when they fit
  const size_t walk_smem = 8 * (size_t)num_bodies;
  if (walk_smem <= kWalkSmemMax) {
    cudaFuncSetAttribute(sis_levels_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)walk_smem);
    sis_levels_kernel<true><<<1, 256, walk_smem, st>>>(body1, body2, d_count, capacity,
                                                      num_bodies, level, last, first,
                                                      iterations, slots, hdr, ctx->d_err);
  } else {
    sis_levels_kernel<false><<<1, 256, 0, st>>>(body1, body2, d_count, capacity, num_bodies,
                                               level, last, first, iterations, slots, hdr,
                                               ctx->d_err);
  }
  sis_sizes_kernel<<<gg, 256, 0, st>>>(level, hdr, run);
  sis_layout_kernel<<<1, kLayoutThreads, 0, st>>>(hdr, run, order);
  sis_pack_kernel<<<gg, 256, 0, st>>>(C, B, geo, level, hdr, run, order, rec, accs);
  // sweeps: the bodies' velocities in shared memory when they fit
  const size_t body_smem = 32 * (size_t)num_bodies;
  const bool shared = body_smem <= kSisSmemMax;
  const size_t smem = shared ? body_smem : 0;
  auto* sweep = shared ? sis_sweep_kernel<true> : sis_sweep_kernel<false>;
  cudaFuncSetAttribute(sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // as many schedules as `capacity` contacts take; with fewer the last ones find no sweeps left
  const int fewest = (int)std::min((long long)iterations, slots / capacity);
  for (int i = 0; i * (long long)fewest < iterations; ++i) {
    sweep<<<1, kSisThreads, smem, st>>>(B, hdr, num_bodies, i, iterations, 100.f, run, rec, accs,
                                        vrel);
    sis_friction_kernel<<<gg, 256, 0, st>>>(C, geo, hdr, order, vrel, i, iterations, accs);
  }
  return arh::check_launch("ar_sequential_impulse");
}

}  // extern "C"
