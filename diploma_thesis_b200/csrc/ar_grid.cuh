// Uniform grid addressing: calcGridPos / calcGridHash (Kernels/particleKernels.cu:150-167,
// RigidBodies/UniformGridDEM.cu:25-41).
#pragma once
#include "ar_internal.cuh"

namespace ar_grid {

struct Grid {
  float ox, oy, oz;     // world origin
  float cx, cy, cz;     // cell edge per axis
  uint32_t gx, gy, gz;  // cells per axis (powers of two)

  static Grid from_params(const ar_sim_params& p) {
    Grid g;
    g.ox = p.world_origin[0]; g.oy = p.world_origin[1]; g.oz = p.world_origin[2];
    g.cx = p.cell_size[0]; g.cy = p.cell_size[1]; g.cz = p.cell_size[2];
    g.gx = p.grid_size[0]; g.gy = p.grid_size[1]; g.gz = p.grid_size[2];
    return g;
  }
  // cell = floor((p - origin) / cell) -- IEEE division, then floorf, then conversion to int
  __host__ __device__ __forceinline__ int3 cell_of(float3 p) const {
    return make_int3((int)floorf((p.x - ox) / cx), (int)floorf((p.y - oy) / cy),
                     (int)floorf((p.z - oz) / cz));
  }
  // wrap with & (G - 1), linearise z-major
  __host__ __device__ __forceinline__ uint32_t hash(int3 c) const {
    const uint32_t x = (uint32_t)c.x & (gx - 1), y = (uint32_t)c.y & (gy - 1),
                   z = (uint32_t)c.z & (gz - 1);
    return z * gy * gx + y * gx + x;
  }
};

// Calls visit(first, end) for every occupied cell among the 27 around `c`, in z, y, x order, with
// its range of sorted slots, and row_done() after every row of three.  The cell starts of a row are loaded one row ahead; empty cells are
// passed over (a float sum that starts at +0 is never -0, so the +0 that an empty cell would add
// changes nothing).  All lanes of a warp look at the same neighbour at a time, so that their
// loads, like their cells, lie side by side: letting each lane jump to its next occupied cell
// scattered the loads and was slower.
template <class Visit, class RowDone>
__device__ __forceinline__ void for_occupied(const Grid& g, int3 c,
                                             const uint32_t* __restrict__ cell_start,
                                             const uint32_t* __restrict__ cell_end, Visit visit,
                                             RowDone row_done) {
  uint32_t x[3], start[3], next[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) x[i] = (uint32_t)(c.x + i - 1) & (g.gx - 1);
  auto row_of = [&](int dz, int dy) {
    return (((uint32_t)(c.z + dz) & (g.gz - 1)) * g.gy + ((uint32_t)(c.y + dy) & (g.gy - 1))) * g.gx;
  };
  uint32_t row = row_of(-1, -1);
#pragma unroll
  for (int i = 0; i < 3; ++i) next[i] = __ldg(cell_start + row + x[i]);
  for (int dz = -1, dy = -1; dz <= 1;) {
    const uint32_t here = row;
#pragma unroll
    for (int i = 0; i < 3; ++i) start[i] = next[i];
    if (++dy > 1) {
      dy = -1;
      ++dz;
    }
    if (dz <= 1) {
      row = row_of(dz, dy);
#pragma unroll
      for (int i = 0; i < 3; ++i) next[i] = __ldg(cell_start + row + x[i]);
    }
    uint32_t end[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) end[i] = start[i] != ar::kEmpty ? __ldg(cell_end + here + x[i]) : 0u;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (start[i] != ar::kEmpty) visit(start[i], end[i]);
    row_done();
  }
}
template <class Visit>
__device__ __forceinline__ void for_occupied(const Grid& g, int3 c,
                                             const uint32_t* __restrict__ cell_start,
                                             const uint32_t* __restrict__ cell_end, Visit visit) {
  for_occupied(g, c, cell_start, cell_end, visit, [] {});
}

}  // namespace ar_grid
