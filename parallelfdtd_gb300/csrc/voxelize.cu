// Solid voxelization of a triangle mesh into the voxelizer's node bytes.
//
// The reference voxelizes with an external library (hakarlss/Voxelizer,
// not vendored, version unpinned; called from
// src/kernels/voxelizationUtils.cu:55-136) whose output is one boundary id
// 0..27 per node (0 solid, 1..8 corners, 9..20 edges, 21..26 faces, 27 air)
// and one material byte.  This file produces the same two arrays on the GPU
// from the room's boundary mesh (closed; closed obstacles inside):
//
//  * grid: node i at lo + (i - 1) dx per axis, lo the mesh's bounding-box
//    minimum, so that a point p of the mesh maps to node ROUND((p - lo)/dx) + 1
//    as the reference's source and receiver coordinates do
//    (SimulationParameters.cpp:200-224); one layer outside the box on every
//    side, so the outermost nodes are solid.  Nodes are sampled a small
//    irrational fraction of dx above their nominal position on every axis, so
//    a node on a wall plane belongs to the side the offset points to;
//  * solid / air: one thread per (x, y) column casts a ray along +z and counts
//    triangle crossings below each node (odd = inside the room = air); the
//    sampling offset keeps the ray off the shared edges of a grid-aligned
//    mesh; the geometry is evaluated in double;
//  * air nodes with solid on both sides of an axis have no boundary id in the
//    voxelizer's table and are made solid, repeatedly until none is left;
//  * materials: a solid node next to air takes the material of the triangle
//    crossed by the segment to its first air neighbour (order -x, +x, -y, +y,
//    -z, +z); a solid node filled in by the previous rule takes its first
//    solid neighbour's material; a boundary node takes the material of its
//    first solid neighbour in the same order, air nodes 0;
//  * ids from the 6-neighbour missing mask with the voxelizer's table.
// These conventions are the ones of parallelfdtd_gb300/rooms.py, so a
// grid-aligned box mesh voxelizes to exactly the procedural room.
#include "common.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace pfdtd {
namespace {

constexpr int kMaxCrossings = 64;   // triangle crossings per column
constexpr int kTriTile = 128;       // triangles staged in shared memory per pass
constexpr int64_t kMostEntries = 32 << 20, kMostCells = 4 << 20;  // of the triangle lists
constexpr int64_t kFewTris = 64, kFewNodes = 1 << 19;  // that are not binned
// sampling offsets (fractions of dx) per axis
constexpr double kEpsX = 1.2345678901e-5, kEpsY = 3.1415926536e-5, kEpsZ = 2.2360679775e-5;

// Missing-neighbour mask (bit set = solid) -> boundary id; 0 where a mask has
// both sides of an axis missing (no id in the voxelizer's table).
__constant__ uint8_t c_bid_lut[64] = {
    27, 24, 25, 0, 22, 20, 19, 0, 23, 18, 17, 0, 0, 0, 0, 0, 26, 16, 15, 0, 14, 8,
    7,  0,  13, 6, 5,  0,  0,  0, 0, 0, 21, 12, 11, 0, 10, 4, 3, 0, 9, 2,  1,  0, 0,
    0,  0,  0,  0, 0,  0,  0,  0, 0, 0, 0,  0,  0,  0, 0, 0, 0, 0, 0};

struct Tri {
  float v[9];      // three vertices
  uint32_t mat;    // material byte
};

__device__ __forceinline__ bool valid_mask(unsigned m) {
  return (m & 3u) != 3u && (m & 12u) != 12u && (m & 48u) != 48u;
}

// Crossing of the line {(a0, a1) fixed, t free} with a triangle, the line's
// free axis `ax` and the two fixed axes (c0, c1): returns true and t when the
// point (a0, a1) lies strictly inside the triangle's projection.
__device__ __forceinline__ bool line_cross(const Tri& t, int ax, int c0, int c1, double a0,
                                           double a1, double* tt) {
  const double x0 = t.v[c0], y0 = t.v[c1], x1 = t.v[3 + c0], y1 = t.v[3 + c1];
  const double x2 = t.v[6 + c0], y2 = t.v[6 + c1];
  const double e0 = (x1 - x0) * (a1 - y0) - (y1 - y0) * (a0 - x0);
  const double e1 = (x2 - x1) * (a1 - y1) - (y2 - y1) * (a0 - x1);
  const double e2 = (x0 - x2) * (a1 - y2) - (y0 - y2) * (a0 - x2);
  const bool in = (e0 > 0 && e1 > 0 && e2 > 0) || (e0 < 0 && e1 < 0 && e2 < 0);
  if (!in) return false;
  const double area = e0 + e1 + e2;
  if (area == 0.0) return false;
  // barycentric weights of vertices 2, 0, 1 are e0, e1, e2 over the area
  *tt = (e1 * t.v[ax] + e2 * t.v[3 + ax] + e0 * t.v[6 + ax]) / area;
  return true;
}

// Whether the point (a0, a1) lies within `margin` of the triangle's bounding
// box in the plane (c0, c1): FP32 comparisons that spare most triangles of a
// list the FP64 test (an SM issues about two FP64 operations a cycle).  The
// margin (box_margin) is a node and more, far above the rounding of the point
// to FP32.
__device__ __forceinline__ bool near_box(const Tri& t, int c0, int c1, float a0, float a1,
                                         float margin) {
  const float x0 = t.v[c0], x1 = t.v[3 + c0], x2 = t.v[6 + c0];
  const float y0 = t.v[c1], y1 = t.v[3 + c1], y2 = t.v[6 + c1];
  return a0 >= fminf(x0, fminf(x1, x2)) - margin && a0 <= fmaxf(x0, fmaxf(x1, x2)) + margin &&
         a1 >= fminf(y0, fminf(y1, y2)) - margin && a1 <= fmaxf(y0, fmaxf(y1, y2)) + margin;
}
__device__ __forceinline__ float box_margin(double a0, double a1, double dx) {
  return (float)dx + 1e-6f * fmaxf(fabsf((float)a0), fabsf((float)a1));
}

// Triangle lists per cell of the voxel grid.  The crossing tests below need
// only the triangles near a column or a node, so every triangle is entered in
// the cells (boxes of `cell` nodes an axis) that its bounding box, widened by
// two nodes on every side, touches: two nodes are far more than the rounding of
// the double-precision tests, so no triangle that passes a test is missing
// from the list.  A list holds its triangles in no particular order; the users
// do not depend on one.
struct Bins {
  int n[3];        // cells per axis
  int cell[3];     // nodes per cell
  double lo[3], inv_dx;
};

// First and last cell that the triangle touches along axis a.
__host__ __device__ inline void cell_range(const Bins& g, const Tri& t, int a, int* c0, int* c1) {
  const double u = t.v[a], v = t.v[3 + a], w = t.v[6 + a];
  const double mn = fmin(u, fmin(v, w)), mx = fmax(u, fmax(v, w));
  // node i lies at lo + (i - 1) dx
  const double i0 = floor((mn - g.lo[a]) * g.inv_dx) - 1.0, i1 = ceil((mx - g.lo[a]) * g.inv_dx) + 3.0;
  const double last = (double)g.n[a] - 1.0;
  *c0 = (int)fmin(fmax(floor(i0 / g.cell[a]), 0.0), last);
  *c1 = (int)fmin(fmax(floor(i1 / g.cell[a]), 0.0), last);
}

// One warp per triangle: counts[cell]++ (list null), or list entries at the
// cell's cursor (cursor = the cell's end offset, counted down).
__global__ void k_bin(const Tri* __restrict__ tris, int64_t nt, Bins g, int* __restrict__ cursor,
                      int* __restrict__ list) {
  const int lane = threadIdx.x & 31;
  for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < nt;
       t += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    int a0, a1, b0, b1, c0, c1;
    cell_range(g, tris[t], 0, &a0, &a1);
    cell_range(g, tris[t], 1, &b0, &b1);
    cell_range(g, tris[t], 2, &c0, &c1);
    const int na = a1 - a0 + 1, nb = b1 - b0 + 1;
    const int64_t n = (int64_t)na * nb * (c1 - c0 + 1);
    for (int64_t k = lane; k < n; k += 32) {
      const int a = a0 + (int)(k % na), b = b0 + (int)(k / na % nb), c = c0 + (int)(k / ((int64_t)na * nb));
      int* at = cursor + ((int64_t)c * g.n[1] + b) * g.n[0] + a;
      if (list) list[atomicSub(at, 1) - 1] = (int)t;
      else atomicAdd(at, 1);
    }
  }
}

// Inclusive prefix sum of the cell counts, one block: begin[c + 1] and the
// fill cursor both receive the end of cell c's list.
__global__ void __launch_bounds__(1024) k_bin_scan(int* __restrict__ cursor, int* __restrict__ begin,
                                                   int64_t n) {
  __shared__ int warp_sum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) {
    carry = 0;
    begin[0] = 0;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = 0; base < n; base += 1024) {
    const int64_t i = base + threadIdx.x;
    int v = i < n ? cursor[i] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) warp_sum[w] = v;
    __syncthreads();
    if (w == 0) {
      int u = warp_sum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int q = __shfl_up_sync(0xffffffffu, u, o);
        if (lane >= o) u += q;
      }
      warp_sum[lane] = u;
    }
    __syncthreads();
    v += carry + (w > 0 ? warp_sum[w - 1] : 0);
    if (i < n) {
      cursor[i] = v;
      begin[i + 1] = v;
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = v;
    __syncthreads();
  }
}

// Column parity: solid[] = 1 outside the room, 0 inside.  A block takes 32 x 4
// columns (a warp writes 32 neighbouring bytes) and the list of the column bin
// that holds them; the crossings it finds are those of a loop over every
// triangle, which took 19 ms on the room of k_surface_mat's note; 0.7 ms now.
__global__ void __launch_bounds__(128) k_parity(const Tri* __restrict__ tris, Bins g,
                         const int* __restrict__ begin, const int* __restrict__ list, int X, int Y,
                         int Z, double lo_x, double lo_y, double lo_z, double dx,
                         uint8_t* __restrict__ solid, int* __restrict__ err) {
  __shared__ Tri st[kTriTile];
  const int tiles_x = (X + 31) / 32, ti = blockIdx.x % tiles_x * 32, tj = blockIdx.x / tiles_x * 4;
  const int bin = tj / g.cell[1] * g.n[0] + ti / g.cell[0];
  const int i = ti + (threadIdx.x & 31), j = tj + (threadIdx.x >> 5);
  const bool active = i < X && j < Y;
  const double px = lo_x + (i - 1 + kEpsX) * dx;
  const double py = lo_y + (j - 1 + kEpsY) * dx;
  double zc[kMaxCrossings];
  const float pxf = (float)px, pyf = (float)py, margin = box_margin(px, py, dx);
  int nc = 0;
  bool overflow = false;
  const int first = begin[bin], end = begin[bin + 1];
  for (int base = first; base < end; base += kTriTile) {
    __syncthreads();
    for (int k = threadIdx.x; k < kTriTile && base + k < end; k += blockDim.x)
      st[k] = tris[list[base + k]];
    __syncthreads();
    const int n = min(end - base, kTriTile);
    if (!active) continue;
    for (int k = 0; k < n; ++k) {
      double t;
      if (near_box(st[k], 0, 1, pxf, pyf, margin) && line_cross(st[k], 2, 0, 1, px, py, &t)) {
        if (nc < kMaxCrossings) zc[nc++] = t;
        else overflow = true;
      }
    }
  }
  if (!active) return;
  if (overflow) atomicExch(err, 1);
  // insertion sort of the crossings along z
  for (int a = 1; a < nc; ++a) {
    const double v = zc[a];
    int b = a - 1;
    while (b >= 0 && zc[b] > v) { zc[b + 1] = zc[b]; --b; }
    zc[b + 1] = v;
  }
  int below = 0;
  for (int k = 0; k < Z; ++k) {
    const double z = lo_z + (k - 1 + kEpsZ) * dx;
    while (below < nc && zc[below] < z) ++below;
    solid[((int64_t)k * Y + j) * X + i] = (below & 1) ? 0 : 1;
  }
}

__device__ __forceinline__ int64_t nb_index(int64_t c, int d, int X, int64_t XY) {
  switch (d) {
    case 0: return c - 1;
    case 1: return c + 1;
    case 2: return c - X;
    case 3: return c + X;
    case 4: return c - XY;
    default: return c + XY;
  }
}

__device__ __forceinline__ bool nb_inside(int x, int y, int z, int d, int X, int Y, int Z) {
  switch (d) {
    case 0: return x > 0;
    case 1: return x < X - 1;
    case 2: return y > 0;
    case 3: return y < Y - 1;
    case 4: return z > 0;
    default: return z < Z - 1;
  }
}

// Missing-neighbour mask of node c (neighbours outside the grid count solid).
__device__ __forceinline__ unsigned missing_mask(const uint8_t* __restrict__ solid, int64_t c,
                                                 int x, int y, int z, int X, int Y, int Z,
                                                 int64_t XY) {
  unsigned m = 0;
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (!nb_inside(x, y, z, d, X, Y, Z) || solid[nb_index(c, d, X, XY)]) m |= 1u << d;
  return m;
}

// Surface materials: a solid node with an air neighbour takes the material
// of the triangle crossed by the segment to its first air neighbour (the
// crossing nearest to the node); 255 when no triangle crosses it.
//
// Each such node tests the triangles of its own cell's list.  With every
// triangle tested for every surface node this kernel took 820 ms on a
// 512 x 384 x 256 room of 1548 triangles (1 M surface nodes, FP64 crossing
// tests); with the lists it takes 2.6 ms (the FP64
// tests of the listed triangles near a node, one at a time).  Ties go to the triangle with the
// lower index, as in a loop over all of them in order.
__global__ void k_surface_mat(const Tri* __restrict__ tris, Bins g, const int* __restrict__ begin,
                              const int* __restrict__ list, const uint8_t* __restrict__ solid,
                              int X, int Y, int Z, double lo_x, double lo_y, double lo_z,
                              double dx, uint8_t* __restrict__ smat) {
  const int64_t XY = (int64_t)X * Y;
  const int tiles_x = (X + 31) / 32;
  const int x = blockIdx.x % tiles_x * 32 + threadIdx.x;
  const int y = blockIdx.x / tiles_x * 4 + threadIdx.y;
  if (x >= X || y >= Y) return;
  const int cxy = (y / g.cell[1]) * g.n[0] + x / g.cell[0];
  for (int z = blockIdx.y; z < Z; z += gridDim.y) {
    const int64_t c = (int64_t)z * XY + (int64_t)y * X + x;
    if (!solid[c]) continue;
    int dir = -1;
    for (int d = 0; d < 6 && dir < 0; ++d)
      if (nb_inside(x, y, z, d, X, Y, Z) && !solid[nb_index(c, d, X, XY)]) dir = d;
    if (dir < 0) continue;
    const int ax = dir >> 1;
    const double sgn = (dir & 1) ? 1.0 : -1.0;
    const double p[3] = {lo_x + (x - 1 + kEpsX) * dx, lo_y + (y - 1 + kEpsY) * dx,
                         lo_z + (z - 1 + kEpsZ) * dx};
    const int c0 = ax == 0 ? 1 : 0, c1 = ax == 2 ? 1 : 2;
    const double a0 = ax == 0 ? p[1] : p[0], a1 = ax == 2 ? p[1] : p[2];
    const double pa = ax == 0 ? p[0] : (ax == 1 ? p[1] : p[2]);
    const int cell = (z / g.cell[2]) * g.n[1] * g.n[0] + cxy;
    const float margin = box_margin(a0, a1, dx);
    double best = 2.0;
    int best_t = -1;
    for (int k = begin[cell]; k < begin[cell + 1]; ++k) {
      const int t = list[k];
      double at;
      if (near_box(tris[t], c0, c1, (float)a0, (float)a1, margin) &&
          line_cross(tris[t], ax, c0, c1, a0, a1, &at)) {
        const double s = (at - pa) * sgn / dx;  // distance along the segment, in voxels
        if (s >= 0.0 && s <= 1.0 && (s < best || (s == best && t < best_t))) {
          best = s;
          best_t = t;
        }
      }
    }
    smat[c] = best_t >= 0 ? (uint8_t)tris[best_t].mat : (uint8_t)255;
  }
}

// One Jacobi pass of the slot closing: air nodes with solid on both sides of
// an axis become solid with their first solid neighbour's material.
__global__ void k_close_slots(const uint8_t* __restrict__ solid, const uint8_t* __restrict__ smat,
                              uint8_t* __restrict__ solid_out, uint8_t* __restrict__ smat_out,
                              int X, int Y, int Z, int* __restrict__ changed) {
  const int64_t XY = (int64_t)X * Y, N = XY * Z;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N;
       c += (int64_t)gridDim.x * blockDim.x) {
    uint8_t s = solid[c], m = smat[c];
    if (!s) {
      const int x = (int)(c % X), y = (int)((c / X) % Y), z = (int)(c / XY);
      const unsigned mk = missing_mask(solid, c, x, y, z, X, Y, Z, XY);
      if (!valid_mask(mk)) {
        s = 1;
        for (int d = 0; d < 6; ++d)
          if (nb_inside(x, y, z, d, X, Y, Z) && solid[nb_index(c, d, X, XY)]) {
            m = smat[nb_index(c, d, X, XY)];
            break;
          }
        *changed = 1;
      }
    }
    solid_out[c] = s;
    smat_out[c] = m;
  }
}

// Boundary ids and materials.
__global__ void k_ids(const uint8_t* __restrict__ solid, const uint8_t* __restrict__ smat, int X,
                      int Y, int Z, uint8_t* __restrict__ bid, uint8_t* __restrict__ mat) {
  const int64_t XY = (int64_t)X * Y, N = XY * Z;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N;
       c += (int64_t)gridDim.x * blockDim.x) {
    if (solid[c]) {
      bid[c] = 0;
      mat[c] = 0;
      continue;
    }
    const int x = (int)(c % X), y = (int)((c / X) % Y), z = (int)(c / XY);
    const unsigned mk = missing_mask(solid, c, x, y, z, X, Y, Z, XY);
    const uint8_t b = c_bid_lut[mk];
    bid[c] = b;
    uint8_t m = 0;
    if (b > 0 && b < 27) {
      for (int d = 0; d < 6; ++d)
        if (nb_inside(x, y, z, d, X, Y, Z) && solid[nb_index(c, d, X, XY)]) {
          m = smat[nb_index(c, d, X, XY)];
          break;
        }
      if (m == 255) m = 0;
    }
    mat[c] = m;
  }
}

// Cells of `cx` x `cy` x `cz` nodes over an X x Y x Z grid.
Bins make_bins(int X, int Y, int Z, int64_t cx, int64_t cy, int64_t cz, const double lo[3], double dx) {
  Bins g;
  const int n[3] = {X, Y, Z};
  const int64_t c[3] = {cx, cy, cz};
  for (int a = 0; a < 3; ++a) {
    g.cell[a] = (int)std::min<int64_t>(c[a], n[a]);
    g.n[a] = (n[a] + g.cell[a] - 1) / g.cell[a];
    g.lo[a] = lo[a];
  }
  g.inv_dx = 1.0 / dx;
  return g;
}

int64_t bin_cells(const Bins& g) { return (int64_t)g.n[0] * g.n[1] * g.n[2]; }

// List entries of all triangles, counting no further than `most`.
int64_t bin_entries(const Bins& g, const std::vector<Tri>& tris, int64_t most) {
  int64_t total = 0;
  for (const Tri& t : tris) {
    int64_t n = 1;
    for (int a = 0; a < 3; ++a) {
      int c0, c1;
      cell_range(g, t, a, &c0, &c1);
      n *= c1 - c0 + 1;
    }
    total += n;
    if (total > most) break;
  }
  return total;
}

// Triangle lists on the device: *begin [cells + 1] and *list, allocated on s.
cudaError_t build_bins(const Tri* d_tris, int64_t nt, const Bins& g, int64_t entries, int** begin,
                       int** list, cudaStream_t s) {
  const int64_t cells = bin_cells(g);
  int* cursor = nullptr;
  cudaError_t e = cudaMallocAsync((void**)begin, sizeof(int) * (cells + 1), s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)list, sizeof(int) * std::max<int64_t>(entries, 1), s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&cursor, sizeof(int) * cells, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(cursor, 0, sizeof(int) * cells, s);
  if (e == cudaSuccess) {
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((nt + 7) / 8, kGridSMs * 8));
    k_bin<<<blocks, 256, 0, s>>>(d_tris, nt, g, cursor, nullptr);
    k_bin_scan<<<1, 1024, 0, s>>>(cursor, *begin, cells);
    k_bin<<<blocks, 256, 0, s>>>(d_tris, nt, g, cursor, *list);
    count_launch(3);
    e = cudaGetLastError();
  }
  if (cursor) cudaFreeAsync(cursor, s);
  return e;
}

int grid_n(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, kGridSMs * 32)); }

}  // namespace
}  // namespace pfdtd

using namespace pfdtd;

extern "C" int pfdtd_voxelize(const float* vertices, int64_t n_vertices, const uint32_t* indices,
                              int64_t n_triangles, const uint8_t* tri_materials,
                              double voxel_edge, int device, uint32_t dims[3], double origin[3],
                              uint8_t* bid_out, uint8_t* mat_out) {
  if (!vertices || !indices || n_vertices < 3 || n_triangles < 1 || !dims)
    return fail(PFDTD_ERR_ARG, "invalid mesh");
  if (!(voxel_edge > 0.0)) return fail(PFDTD_ERR_ARG, "voxel edge must be positive");
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int64_t v = 0; v < n_vertices; ++v)
    for (int a = 0; a < 3; ++a) {
      const double c = vertices[3 * v + a];
      if (!(c == c)) return fail(PFDTD_ERR_ARG, "vertex coordinate is NaN");
      lo[a] = std::min(lo[a], c);
      hi[a] = std::max(hi[a], c);
    }
  // last inside node: the largest i with (i - 1 + eps) dx < extent; one
  // outside layer beyond it
  int64_t n[3];
  const double eps[3] = {kEpsX, kEpsY, kEpsZ};
  for (int a = 0; a < 3; ++a) {
    n[a] = (int64_t)std::floor((hi[a] - lo[a]) / voxel_edge - eps[a]) + 3;
    if (n[a] < 3) n[a] = 3;
  }
  if (n[0] > (1 << 20) || n[1] > (1 << 20) || n[2] > (1 << 20) ||
      n[0] * n[1] * n[2] > ((int64_t)1 << 36))
    return fail(PFDTD_ERR_ARG, "voxel grid too large");
  for (int a = 0; a < 3; ++a) dims[a] = (uint32_t)n[a];
  if (origin)
    for (int a = 0; a < 3; ++a) origin[a] = lo[a] - voxel_edge;  // position of node 0
  if (!bid_out && !mat_out) return PFDTD_OK;
  if (!bid_out || !mat_out) return fail(PFDTD_ERR_ARG, "both output arrays are needed");
  std::vector<Tri> tris((size_t)n_triangles);
  for (int64_t t = 0; t < n_triangles; ++t) {
    for (int k = 0; k < 3; ++k) {
      const uint32_t vi = indices[3 * t + k];
      if ((int64_t)vi >= n_vertices) return fail(PFDTD_ERR_ARG, "triangle index out of range");
      for (int a = 0; a < 3; ++a) tris[t].v[3 * k + a] = vertices[3 * (int64_t)vi + a];
    }
    tris[t].mat = tri_materials ? tri_materials[t] : 0;
  }
  const int X = (int)n[0], Y = (int)n[1], Z = (int)n[2];
  const int64_t N = (int64_t)X * Y * Z;
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  struct Restore {
    int p;
    ~Restore() { if (p >= 0) cudaSetDevice(p); }
  } restore{prev};
  // Column bins of k_parity's block tiles and node cells of 8^3; both larger (up
  // to the whole grid, which is the loop over every triangle) where a few large
  // triangles or a huge grid would make the lists or the cell table too long.  A
  // few triangles in a small grid are one cell of each kind from the start, whose
  // list goes up behind the triangles: binning 12 took 75 us of the 399 of a box of
  // 18^3 nodes.  A call, us, in one cell / binned: 18^3 320 / 399, 66^3 450 / 490, but
  // 130^3 1300 / 1220, 258^3 4400 / 3750.
  Bins gc, gn;
  int64_t ec = n_triangles, en = n_triangles;
  const bool few = n_triangles <= kFewTris && N <= kFewNodes;
  if (few) {
    gc = gn = make_bins(X, Y, Z, X, Y, Z, lo, voxel_edge);
    std::vector<int> one(2 + (size_t)n_triangles);
    one[0] = 0;
    one[1] = (int)n_triangles;
    for (int t = 0; t < (int)n_triangles; ++t) one[2 + t] = t;
    const size_t bytes = sizeof(int) * one.size();
    tris.resize((size_t)n_triangles + (bytes + sizeof(Tri) - 1) / sizeof(Tri));
    std::memcpy((void*)(tris.data() + n_triangles), one.data(), bytes);
  } else {
    for (int64_t m = 1;; m *= 2) {
      gc = make_bins(X, Y, Z, 32 * m, 4 * m, Z, lo, voxel_edge);
      ec = bin_entries(gc, tris, kMostEntries);
      if ((ec <= kMostEntries && bin_cells(gc) <= kMostCells) || bin_cells(gc) == 1) break;
    }
    for (int64_t c = 8;; c *= 2) {
      gn = make_bins(X, Y, Z, c, c, c, lo, voxel_edge);
      en = bin_entries(gn, tris, kMostEntries);
      if ((en <= kMostEntries && bin_cells(gn) <= kMostCells) || bin_cells(gn) == 1) break;
    }
    if (bin_cells(gc) == 1) ec = n_triangles;
    if (bin_cells(gn) == 1) en = n_triangles;
  }
  cudaStream_t s = nullptr;
  PFDTD_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  Tri* d_tris = nullptr;
  uint8_t *d_solid = nullptr, *d_smat = nullptr, *d_s2 = nullptr, *d_m2 = nullptr;
  int* d_flags = nullptr;  // [0] overflow, [1] changed
  cudaError_t e = cudaMallocAsync((void**)&d_tris, sizeof(Tri) * tris.size(), s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_solid, N, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_smat, N, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_s2, N, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_m2, N, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_flags, 2 * sizeof(int), s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_tris, tris.data(), sizeof(Tri) * tris.size(), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_flags, 0, 2 * sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_smat, 255, N, s);
  int flags[2] = {0, 0};
  int *bc = nullptr, *lc = nullptr, *bn = nullptr, *ln = nullptr;
  if (n_triangles >= INT32_MAX) e = cudaErrorInvalidValue;  // triangle numbers are ints here
  if (few) {
    bc = bn = (int*)(d_tris + n_triangles);
    lc = ln = bc + 2;
  } else {
    if (e == cudaSuccess) e = build_bins(d_tris, n_triangles, gc, ec, &bc, &lc, s);
    if (e == cudaSuccess) e = build_bins(d_tris, n_triangles, gn, en, &bn, &ln, s);
  }
  if (e == cudaSuccess) {
    const int64_t tiles = (int64_t)((X + 31) / 32) * ((Y + 3) / 4);
    k_parity<<<(unsigned)tiles, 128, 0, s>>>(d_tris, gc, bc, lc, X, Y, Z, lo[0], lo[1], lo[2],
                                                     voxel_edge, d_solid, d_flags);
    count_launch();
    k_surface_mat<<<dim3((unsigned)tiles, std::min(Z, 65535)), dim3(32, 4), 0, s>>>(
        d_tris, gn, bn, ln, d_solid, X, Y, Z, lo[0], lo[1], lo[2], voxel_edge, d_smat);
    count_launch();
    e = cudaGetLastError();
  }
  // close slots until none is left (each pass ping-pongs the two buffers)
  for (int pass = 0; e == cudaSuccess && pass < 4096; ++pass) {
    e = cudaMemsetAsync(d_flags + 1, 0, sizeof(int), s);
    if (e != cudaSuccess) break;
    k_close_slots<<<grid_n(N), 256, 0, s>>>(d_solid, d_smat, d_s2, d_m2, X, Y, Z, d_flags + 1);
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(flags, d_flags, sizeof(flags), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    std::swap(d_solid, d_s2);
    std::swap(d_smat, d_m2);
    if (e != cudaSuccess || !flags[1]) break;
  }
  if (e == cudaSuccess) {
    k_ids<<<grid_n(N), 256, 0, s>>>(d_solid, d_smat, X, Y, Z, d_s2, d_m2);
    count_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(bid_out, d_s2, N, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(mat_out, d_m2, N, cudaMemcpyDeviceToHost, s);
  if (few) bc = lc = bn = ln = nullptr;  // part of d_tris
  for (void* p : {(void*)d_tris, (void*)d_solid, (void*)d_smat, (void*)d_s2, (void*)d_m2,
                  (void*)d_flags, (void*)bc, (void*)lc, (void*)bn, (void*)ln})
    if (p) cudaFreeAsync(p, s);
  const cudaError_t e2 = cudaStreamSynchronize(s);
  cudaStreamDestroy(s);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return cuda_fail(e, "voxelization", __FILE__, __LINE__);
  if (flags[0]) return fail(PFDTD_ERR_UNSUPPORTED, "more than 64 surface crossings in a column");
  return PFDTD_OK;
}
