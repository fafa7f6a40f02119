// Marching-cubes surface of the density field: Particles::getSurfacePrims
// (particles.cpp:352-385) with generateGridCell (:309-323), getVertexNormal (:399-412),
// estimateDensityAt (:446-453) and polygonise / vertexInterp (marching.cpp).
//
//   k_surf_cells    cells with a particle in their 27 cells
//   k_surf_density  the field at every grid corner (one evaluation per corner; the
//                   reference evaluates each cube's 8 corners separately, at the same
//                   points up to the last bit of x1 + step)
//   k_surf_count    cube index (bit k set when corner k is below the iso level) and its
//                   triangle count, scanned within tiles of kCubeTile cubes; k_surf_tiles
//                   scans the tiles' sums
//   k_surf_vertices edge vertices (vertexInterp), triangles in cube order; each grid edge
//                   into a table
//   k_surf_vnormals a normal per grid edge, from central differences of the field at
//                   +-0.001; k_surf_normals hands them to the triangles
//
// Cubes are visited in the reference's loop order (x outer, then y, then z) and
// corners and edges are numbered as in generateGridCell and polygonise, so the
// vertices and their order follow the reference. The triangulation of each cube
// configuration is this library's own table (built by build_table below): on a
// face with four crossing edges the segments cut off the corners below the iso
// level, the segments of the six faces close into loops, and each loop is a fan
// from the first of its vertices that shares no face with a non-adjacent vertex of
// the loop. The surface is closed across cubes.
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "pbf_device.cuh"

namespace pbf {

namespace {

// corner k of a cube, as generateGridCell lays it out: (x, y, z) in {0, 1}
constexpr int kCorner[8][3] = {{0, 0, 0}, {0, 1, 0}, {1, 1, 0}, {1, 0, 0},
                               {0, 0, 1}, {0, 1, 1}, {1, 1, 1}, {1, 0, 1}};
// edge e joins corners kEdge[e][0] and kEdge[e][1], as polygonise numbers them
constexpr int kEdge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                              {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

int edge_between(int a, int b) {
  for (int e = 0; e < 12; ++e)
    if ((kEdge[e][0] == a && kEdge[e][1] == b) || (kEdge[e][0] == b && kEdge[e][1] == a)) return e;
  return -1;
}

}  // namespace

void build_table(SurfTable* t) {
  std::memset(t, 0, sizeof(*t));
  // the six faces as corner cycles (corners of a face in order around it)
  int face[6][4];
  int nf = 0;
  for (int axis = 0; axis < 3; ++axis) {
    for (int side = 0; side < 2; ++side) {
      const int u = (axis + 1) % 3, v = (axis + 2) % 3;
      // corners of this face in the cycle (0,0) (1,0) (1,1) (0,1) of (u, v)
      const int cyc[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
      for (int k = 0; k < 4; ++k) {
        for (int c = 0; c < 8; ++c) {
          if (kCorner[c][axis] == side && kCorner[c][u] == cyc[k][0] && kCorner[c][v] == cyc[k][1]) face[nf][k] = c;
        }
      }
      ++nf;
    }
  }
  auto same_face = [&](int ea, int eb) {
    for (int f = 0; f < 6; ++f) {
      bool a = false, b = false;
      for (int k = 0; k < 4; ++k) {
        const int e = edge_between(face[f][k], face[f][(k + 1) % 4]);
        a |= e == ea;
        b |= e == eb;
      }
      if (a && b) return true;
    }
    return false;
  };
  for (int ci = 0; ci < 256; ++ci) {
    bool in[8];
    for (int c = 0; c < 8; ++c) in[c] = (ci >> c) & 1;
    uint16_t mask = 0;
    for (int e = 0; e < 12; ++e)
      if (in[kEdge[e][0]] != in[kEdge[e][1]]) mask |= static_cast<uint16_t>(1u << e);
    t->edges[ci] = mask;
    // face segments: partner[e][0..1] = the edges joined to e on its two faces
    int partner[12][2], np[12] = {};
    for (int f = 0; f < 6; ++f) {
      int es[4], cross[4], nc = 0;
      for (int k = 0; k < 4; ++k) {
        es[k] = edge_between(face[f][k], face[f][(k + 1) % 4]);
        if (in[face[f][k]] != in[face[f][(k + 1) % 4]]) cross[nc++] = k;
      }
      auto join = [&](int a, int b) {
        partner[a][np[a]++] = b;
        partner[b][np[b]++] = a;
      };
      if (nc == 2) {
        join(es[cross[0]], es[cross[1]]);
      } else if (nc == 4) {  // cut off the corners below the iso level
        for (int k = 0; k < 4; ++k)
          if (in[face[f][k]]) join(es[(k + 3) % 4], es[k]);
      }
    }
    // loops, from the lowest unused edge, and their fans
    bool used[12] = {};
    int ntri = 0;
    for (int start = 0; start < 12; ++start) {
      if (!(mask & (1u << start)) || used[start]) continue;
      int loop[12], k = 0, prev = -1, cur = start;
      for (;;) {
        loop[k++] = cur;
        used[cur] = true;
        const int next = (prev < 0 || partner[cur][0] != prev) ? partner[cur][0] : partner[cur][1];
        prev = cur;
        cur = next;
        if (cur == start) break;
      }
      int apex = 0;
      for (int a = 0; a < k; ++a) {
        bool ok = true;
        for (int i = 2; i < k - 1 && ok; ++i) ok = !same_face(loop[a], loop[(a + i) % k]);
        if (ok) {
          apex = a;
          break;
        }
      }
      for (int i = 1; i < k - 1; ++i) {
        t->tri[ci][3 * ntri] = static_cast<int8_t>(loop[apex]);
        t->tri[ci][3 * ntri + 1] = static_cast<int8_t>(loop[(apex + i) % k]);
        t->tri[ci][3 * ntri + 2] = static_cast<int8_t>(loop[(apex + i + 1) % k]);
        ++ntri;
      }
    }
    t->ntri[ci] = static_cast<uint8_t>(ntri);
  }
}

const SurfTable& surf_table() {
  static SurfTable table;
  static std::once_flag once;
  std::call_once(once, [] { build_table(&table); });
  return table;
}

namespace {

constexpr uint32_t kCubeTile = 2048;  // cubes of a block of k_surf_count

// kCorner / kEdge for device code: corner k has x = 1 for k in {2, 3, 6, 7}, y = 1 for
// k in {1, 2, 5, 6}, z = k / 4; edge e < 8 joins e and (e & 4) | ((e + 1) & 3), edge e >= 8
// joins e - 8 and e - 4
__device__ __forceinline__ int corner_x(int k) { return (0xCC >> k) & 1; }
__device__ __forceinline__ int corner_y(int k) { return (0x66 >> k) & 1; }
__device__ __forceinline__ int corner_z(int k) { return k >> 2; }
__device__ __forceinline__ int edge_a(int e) { return e < 8 ? e : e - 8; }
__device__ __forceinline__ int edge_b(int e) { return e < 8 ? ((e & 4) | ((e + 1) & 3)) : e - 4; }

// x1 = min(lo + i step, hi) per axis, computed in FP64 as the reference computes it (on
// the host, SurfGrid::axis)
__device__ __forceinline__ float3 corner_point(const SurfGrid& g, int i, int j, int k) {
  return make_float3(__ldg(&g.axis[i]), __ldg(&g.axis[g.nc[0] + 1 + j]), __ldg(&g.axis[g.nc[0] + g.nc[1] + 2 + k]));
}

// any[c]: a particle lies in one of the 27 cells around cell c. Most corners of a surface grid
// see none (3 of 4 over a box a quarter full), and leave k_surf_density after one byte.
__global__ void k_surf_cells(const uint32_t* __restrict__ cell_start, const SceneDesc* __restrict__ scenes,
                             uint8_t* __restrict__ any, uint32_t m) {
  chain_begin();
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  const SceneDesc& sc = scenes[0];
  const int dx = sc.dim[0], dy = sc.dim[1], dz = sc.dim[2];
  const int x = static_cast<int>(c % dx), y = static_cast<int>((c / dx) % dy), z = static_cast<int>(c / dx / dy);
  const int x0 = max(x - 1, 0), x1 = min(x + 1, dx - 1);
  bool some = false;
  for (int k = max(z - 1, 0); k <= min(z + 1, dz - 1); ++k)
    for (int j = max(y - 1, 0); j <= min(y + 1, dy - 1); ++j) {
      const uint32_t row = static_cast<uint32_t>((k * dy + j) * dx);
      some |= __ldg(&cell_start[row + x0]) != __ldg(&cell_start[row + x1 + 1]);
    }
  any[c] = some ? 1 : 0;
}

// Whether the lanes of a box [lo, hi] walk the rows around all of it (density_together), or each
// lane those around its own point: a wide box holds many candidates that are near few of its
// points, and each lane would read all of them. A surface of 1M particles with cubes of h (a box of
// 1 cell): 250 us together, 290 each; cubes of 1.5 h 257 and 189, 2 h 281 and 171, 4 h 485 and 168,
// 40 h 18,900 and 97.
constexpr float kTogetherCells = 1.25f;
__device__ __forceinline__ bool walk_together(const float3 lo, const float3 hi, const SceneDesc& sc,
                                              const DevParams& P) {
  const float w = fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z) * P.inv_cell;
  return w <= kTogetherCells && in_grid(lo, sc, P.inv_cell) && in_grid(hi, sc, P.inv_cell);
}

// The field, z fastest (the cubes' loop order, so the passes over the cubes read it in lines). 8
// lanes take a block of 2 x 2 x 2 corners and walk its candidates together: with a candidate list
// of its own per lane the pass is bound by the L1 data pipe (a load of 32 lanes touches about 20
// lines), with shared ones a load is 4 broadcasts. A warp takes 4 such blocks along z and writes
// whole sectors. 1M particles, 4.25M corners: 381 -> 240 us (274 with two corners a lane).
__global__ void __launch_bounds__(128) k_surf_density(const float4* __restrict__ pos,
                                                      const uint32_t* __restrict__ cell_start,
                                                      const SceneDesc* __restrict__ scenes,
                                                      const uint8_t* __restrict__ any, SurfGrid g,
                                                      float* __restrict__ field, DevParams P) {
  chain_begin();
  const int nx = g.nc[0] + 1, ny = g.nc[1] + 1, nz = g.nc[2] + 1;
  const int lane = static_cast<int>(lane_id()), warp = static_cast<int>(threadIdx.x >> 5);
  const int bx = (nx + 1) / 2, by = (ny + 7) / 8;
  const int b = static_cast<int>(blockIdx.x);
  const int i0 = 2 * (b % bx), j0 = 8 * ((b / bx) % by) + 2 * warp, k0 = 8 * (b / bx / by) + 2 * (lane >> 3);
  const int i = i0 + ((lane >> 2) & 1), j = j0 + ((lane >> 1) & 1), k = k0 + (lane & 1);
  const SceneDesc& sc = scenes[0];
  const bool live = i < nx && j < ny && k < nz;
  const float3 lo = corner_point(g, min(i0, nx - 1), min(j0, ny - 1), min(k0, nz - 1));
  const float3 hi = corner_point(g, min(i0 + 1, nx - 1), min(j0 + 1, ny - 1), min(k0 + 1, nz - 1));
  const float3 p = corner_point(g, min(i, nx - 1), min(j, ny - 1), min(k, nz - 1));
  const bool near = live && any[cell_key(cell_of(p, sc, P.inv_cell), sc)] != 0;
  float v = 0.f;
  if ((__ballot_sync(0xffffffffu, near) >> (lane & 24)) & 0xffu) {
    if (walk_together(lo, hi, sc, P))
      v = P.poly6_c * density_together(p, lo, hi, pos, cell_start, sc, P);
    else if (near)
      v = density_at_point(p, pos, cell_start, sc, P);
  }
  if (live) field[(static_cast<uint32_t>(i) * ny + j) * nz + k] = v;
}

// cube c in the reference's loop order: c = (ix * nc_y + iy) * nc_z + iz (at most 2e9 cubes)
__device__ __forceinline__ void cube_of(const SurfGrid& g, uint32_t c, int* ix, int* iy, int* iz) {
  const uint32_t ny = g.nc[1], nz = g.nc[2], col = c / nz;
  *iz = static_cast<int>(c - col * nz);
  *ix = static_cast<int>(col / ny);
  *iy = static_cast<int>(col - static_cast<uint32_t>(*ix) * ny);
}

__device__ __forceinline__ float corner_value(const float* __restrict__ field, const SurfGrid& g, int i, int j,
                                              int k) {
  return field[(static_cast<uint32_t>(i) * (g.nc[1] + 1) + j) * (g.nc[2] + 1) + k];
}

__device__ __forceinline__ int cube_index(const float* __restrict__ field, const SurfGrid& g, float iso, int ix,
                                          int iy, int iz) {
  int ci = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (corner_value(field, g, ix + corner_x(k), iy + corner_y(k), iz + corner_z(k)) < iso) ci |= 1 << k;
  return ci;
}

__device__ __forceinline__ uint32_t warp_scan(uint32_t v) {  // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane_id() >= static_cast<unsigned>(o)) v += y;
  }
  return v;
}

// first[c]: triangles of the cubes before c in its tile; tile[t]: triangles of tile t. A thread
// takes 4 cubes in a row, a block one tile.
__global__ void __launch_bounds__(kCubeTile / 4) k_surf_count(const float* __restrict__ field,
                                                              const SurfTable* __restrict__ tab, SurfGrid g,
                                                              float iso, uint32_t* __restrict__ first,
                                                              uint32_t* __restrict__ tile, uint32_t ncubes) {
  chain_begin();
  __shared__ uint8_t ntri[256];
  __shared__ uint32_t sums[kCubeTile / 128];
  for (unsigned k = threadIdx.x; k < 256; k += blockDim.x) ntri[k] = tab->ntri[k];
  __syncthreads();
  const uint32_t base = blockIdx.x * kCubeTile + 4 * threadIdx.x;
  uint32_t v[4], s = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    v[u] = 0;
    if (base + u < ncubes) {
      int ix, iy, iz;
      cube_of(g, base + u, &ix, &iy, &iz);
      v[u] = ntri[cube_index(field, g, iso, ix, iy, iz)];
    }
    s += v[u];
  }
  const uint32_t incl = warp_scan(s);
  const unsigned warp = threadIdx.x >> 5;
  if (lane_id() == 31) sums[warp] = incl;
  __syncthreads();
  uint32_t off = incl - s;
  for (unsigned w = 0; w < warp; ++w) off += sums[w];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (base + u < ncubes) first[base + u] = off;
    off += v[u];
  }
  if (threadIdx.x == blockDim.x - 1) tile[blockIdx.x] = off;
}

// Exclusive scan of the tiles' sums in place; tile[tiles] = the total.
__global__ void __launch_bounds__(1024) k_surf_tiles(uint32_t* __restrict__ tile, uint32_t tiles) {
  chain_begin();
  __shared__ uint32_t sums[32];
  uint32_t carry = 0;
  for (uint32_t b = 0; b < tiles; b += 4 * blockDim.x) {
    uint32_t v[4], s = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t at = b + 4 * threadIdx.x + u;
      v[u] = at < tiles ? tile[at] : 0u;
      s += v[u];
    }
    const uint32_t incl = warp_scan(s);
    if (lane_id() == 31) sums[threadIdx.x >> 5] = incl;
    __syncthreads();
    if (threadIdx.x < 32) sums[threadIdx.x] = warp_scan(sums[threadIdx.x]);
    __syncthreads();
    uint32_t off = carry + incl - s + (threadIdx.x < 32 ? 0u : sums[(threadIdx.x >> 5) - 1]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t at = b + 4 * threadIdx.x + u;
      if (at < tiles) tile[at] = off;
      off += v[u];
    }
    carry += sums[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) tile[tiles] = carry;
}

// vertexInterp (marching.cpp): the iso crossing on the edge p1 -> p2
__device__ __forceinline__ float3 vertex_interp(float iso, float3 p1, float3 p2, float v1, float v2) {
  if (fabsf(iso - v1) < 0.00001f) return p1;
  if (fabsf(iso - v2) < 0.00001f) return p2;
  if (fabsf(v1 - v2) < 0.00001f) return p1;
  const float mu = (iso - v1) / (v2 - v1);
  return make_float3(p1.x + mu * (p2.x - p1.x), p1.y + mu * (p2.y - p1.y), p1.z + mu * (p2.z - p1.z));
}

// Triangle t lies in the cube c with first[c] <= t < first[c + 1] (binary search over the tiles,
// then over the tile's cubes; empty cubes have first[c] == first[c + 1]), as the q-th of its cube's
// triangles; its vertex v sits on cube edge e between corners a and b (the cube's own corner order).
struct TriVertex {
  int ix, iy, iz, a, b;
};
__device__ __forceinline__ TriVertex tri_vertex(const float* __restrict__ field, const SurfTable* __restrict__ tab,
                                                const SurfGrid& g, float iso, const uint32_t* __restrict__ first,
                                                const uint32_t* __restrict__ tile, uint32_t ncubes, uint32_t t,
                                                int v) {
  uint32_t lo = 0, hi = (ncubes + kCubeTile - 1) / kCubeTile;  // tile[lo] <= t < tile[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&tile[mid]) <= t) lo = mid;
    else hi = mid;
  }
  const uint32_t rest = t - __ldg(&tile[lo]);
  lo *= kCubeTile;
  hi = min(lo + kCubeTile, ncubes);  // first[lo] <= rest, the tile holds more than rest
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&first[mid]) <= rest) lo = mid;
    else hi = mid;
  }
  TriVertex r;
  cube_of(g, lo, &r.ix, &r.iy, &r.iz);
  const int ci = cube_index(field, g, iso, r.ix, r.iy, r.iz);
  const int e = tab->tri[ci][3 * static_cast<int>(rest - __ldg(&first[lo])) + v];
  r.a = edge_a(e);
  r.b = edge_b(e);
  return r;
}

// The grid edge of a cube edge, independent of the cube: 3 * (index of its lower corner)
// + its axis.
__device__ __forceinline__ unsigned long long edge_key(const SurfGrid& g, const TriVertex& r) {
  const int i = r.ix + min(corner_x(r.a), corner_x(r.b)), j = r.iy + min(corner_y(r.a), corner_y(r.b)),
            k = r.iz + min(corner_z(r.a), corner_z(r.b));
  const int axis = corner_x(r.a) != corner_x(r.b) ? 0 : (corner_y(r.a) != corner_y(r.b) ? 1 : 2);
  const unsigned long long corner =
      (static_cast<unsigned long long>(k) * (g.nc[1] + 1) + j) * static_cast<unsigned long long>(g.nc[0] + 1) + i;
  return 3ull * corner + static_cast<unsigned long long>(axis);
}

constexpr unsigned long long kNoKey = ~0ull;

__device__ __forceinline__ uint32_t key_hash(unsigned long long k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  return static_cast<uint32_t>(k);
}

// One thread per triangle vertex: the vertex's grid edge goes into an open-addressing table
// (linear probing, compare-and-swap; the table holds at least twice the vertices, so a probe
// ends) and the vertex keeps its slot. Vertices shared by the triangles around an edge get
// one slot, so each normal is evaluated once; the thread that filled a slot lists it in
// ulist (warp-aggregated count in *ucount), so that the normals are computed by a dense grid. The
// vertex itself is written here: by vertexInterp on its cube's edge in the cube's own corner order
// (as the reference computes it per cube). A thread per cube instead would leave most lanes of a
// warp on empty cubes while one lane did up to 5 triangles.
__global__ void k_surf_vertices(const float* __restrict__ field, const SurfTable* __restrict__ tab, SurfGrid g,
                                float iso, const uint32_t* __restrict__ first, const uint32_t* __restrict__ tile,
                                uint32_t count, uint32_t ncubes, unsigned long long* keys, uint32_t cap_mask,
                                uint32_t* __restrict__ vslot, uint32_t* __restrict__ ulist, uint32_t* ucount,
                                float* __restrict__ xyz) {
  chain_begin();
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= 3u * count) return;
  const TriVertex r = tri_vertex(field, tab, g, iso, first, tile, ncubes, tid / 3u, static_cast<int>(tid % 3u));
  const int ia = r.ix + corner_x(r.a), ja = r.iy + corner_y(r.a), ka = r.iz + corner_z(r.a);
  const int ib = r.ix + corner_x(r.b), jb = r.iy + corner_y(r.b), kb = r.iz + corner_z(r.b);
  const float3 x = vertex_interp(iso, corner_point(g, ia, ja, ka), corner_point(g, ib, jb, kb),
                                 corner_value(field, g, ia, ja, ka), corner_value(field, g, ib, jb, kb));
  float* o = xyz + 3 * static_cast<size_t>(tid);
  o[0] = x.x;
  o[1] = x.y;
  o[2] = x.z;
  const unsigned long long key = edge_key(g, r);
  uint32_t h = key_hash(key) & cap_mask;
  bool fresh = false;
  for (uint32_t probe = 0; probe <= cap_mask; ++probe) {
    const unsigned long long prev = atomicCAS(&keys[h], kNoKey, key);
    if (prev == kNoKey || prev == key) {
      fresh = prev == kNoKey;
      break;
    }
    h = (h + 1) & cap_mask;
  }
  vslot[tid] = h;
  const unsigned act = __activemask();
  const unsigned m = __ballot_sync(act, fresh);
  if (m) {
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (static_cast<int>(threadIdx.x & 31u) == leader) base = atomicAdd(ucount, static_cast<uint32_t>(__popc(m)));
    base = __shfl_sync(act, base, leader);
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (fresh) ulist[base + __popc(m & lt)] = h;
  }
}

// The normals of the filled table slots (ulist[0, *ucount)): getVertexNormal, normalized central
// differences of estimateDensityAt at +-GRADIENT_EPS around the slot's edge vertex, the vertex taken
// by vertexInterp from the edge's lower corner to its upper corner. 8 lanes take a slot: 6 of them
// its 6 points, walking their candidates together.
__global__ void __launch_bounds__(128) k_surf_vnormals(const float* __restrict__ field, SurfGrid g, float iso,
                                                       const unsigned long long* __restrict__ keys,
                                                       const uint32_t* __restrict__ ulist,
                                                       const uint32_t* __restrict__ ucount,
                                                       float4* __restrict__ nslot, const float4* __restrict__ pos,
                                                       const uint32_t* __restrict__ cell_start,
                                                       const SceneDesc* __restrict__ scenes, DevParams P) {
  chain_begin();
  const uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if ((u & ~3u) >= *ucount) return;  // none of the warp's 4 slots
  const int lane = static_cast<int>(lane_id());
  const uint32_t sidx = ulist[min(u, *ucount - 1)];
  const unsigned long long key = keys[sidx];
  const int axis = static_cast<int>(key % 3ull);
  unsigned long long c = key / 3ull;
  const int nx = g.nc[0] + 1, ny = g.nc[1] + 1;
  const int i = static_cast<int>(c % nx);
  c /= nx;
  const int j = static_cast<int>(c % ny), k = static_cast<int>(c / ny);
  const int i2 = i + (axis == 0), j2 = j + (axis == 1), k2 = k + (axis == 2);
  const float3 x = vertex_interp(iso, corner_point(g, i, j, k), corner_point(g, i2, j2, k2),
                                 corner_value(field, g, i, j, k), corner_value(field, g, i2, j2, k2));
  const float eps = 0.001f;  // GRADIENT_EPS, particles.cpp:16
  const float3 lo = make_float3(x.x - eps, x.y - eps, x.z - eps), hi = make_float3(x.x + eps, x.y + eps, x.z + eps);
  const int q = min(lane & 7, 5);  // point q: axis q / 2, below or above
  float3 p = x;
  set3(p, q >> 1, (q & 1) ? cmp3(hi, q >> 1) : cmp3(lo, q >> 1));
  const SceneDesc& sc = scenes[0];
  const float v = walk_together(lo, hi, sc, P) ? density_together(p, lo, hi, pos, cell_start, sc, P)
                                               : density_sum_at(p, pos, cell_start, sc, P);
  __syncwarp();
  // lanes 0, 2, 4: the density below less the one above, the former not rounded first
  const float d = __fmaf_rn(P.poly6_c, v, -__fmul_rn(P.poly6_c, __shfl_down_sync(0xffffffffu, v, 1)));
  float3 n;
  n.x = __shfl_sync(0xffffffffu, d, 0, 8);
  n.y = __shfl_sync(0xffffffffu, d, 2, 8);
  n.z = __shfl_sync(0xffffffffu, d, 4, 8);
  if ((lane & 7) != 0 || u >= *ucount) return;
  const float nn = sqrtf(dot3(n, n));
  if (nn > 0.f) n = n * (1.0f / nn);
  nslot[sidx] = make_float4(n.x, n.y, n.z, 0.f);
}

__global__ void k_surf_normals(const uint32_t* __restrict__ vslot, const float4* __restrict__ nslot,
                               float* __restrict__ nrm, uint32_t verts) {
  chain_begin();
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= verts) return;
  const float4 n = nslot[vslot[tid]];
  float* m = nrm + 3 * static_cast<size_t>(tid);
  m[0] = n.x;
  m[1] = n.y;
  m[2] = n.z;
}

inline unsigned blocks_for(int64_t n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

}  // namespace

uint32_t surface_tiles(uint32_t cubes) { return (cubes + kCubeTile - 1) / kCubeTile; }

cudaError_t launch_surface_count(const Buffers& b, const DevParams& P, int cur, const SurfGrid& g, float iso,
                                 const SurfTable* tab, uint8_t* any, float* field, uint32_t* first, uint32_t* tile,
                                 cudaStream_t s) {
  const uint32_t cubes = static_cast<uint32_t>(g.nc[0]) * g.nc[1] * g.nc[2];
  const int64_t blocks = static_cast<int64_t>((g.nc[0] + 2) / 2) * ((g.nc[1] + 8) / 8) * ((g.nc[2] + 8) / 8);
  chain_launch(k_surf_cells, blocks_for(b.n_cells, 256), 256, 0, s, b.cell_start, b.scenes, any, b.n_cells);
  chain_launch(k_surf_density, static_cast<unsigned>(blocks), 128, 0, s, b.pos[cur], b.cell_start, b.scenes, any, g,
               field, P);
  chain_launch(k_surf_count, surface_tiles(cubes), kCubeTile / 4, 0, s, field, tab, g, iso, first, tile, cubes);
  chain_launch(k_surf_tiles, 1, 1024, 0, s, tile, surface_tiles(cubes));
  return cudaGetLastError();
}

uint32_t surface_hash_slots(uint32_t triangles) {
  uint32_t c = 1024;
  while (c < 6ull * triangles && c < (1u << 31)) c <<= 1;
  return c;
}

cudaError_t launch_surface_emit(const Buffers& b, const DevParams& P, int cur, const SurfGrid& g, float iso,
                                const SurfTable* tab, const float* field, const uint32_t* first,
                                const uint32_t* tile, float* xyz, float* nrm, uint32_t cap, const SurfHash& hs,
                                cudaStream_t s) {
  const uint32_t cubes = static_cast<uint32_t>(g.nc[0]) * g.nc[1] * g.nc[2];
  if (cap == 0) return cudaSuccess;
  const uint32_t slots = surface_hash_slots(cap);
  cudaError_t e = cudaMemsetAsync(hs.keys, 0xff, sizeof(unsigned long long) * slots, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(hs.ucount, 0, sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  const uint32_t verts = 3 * cap;
  chain_launch(k_surf_vertices, blocks_for(verts, 128), 128, 0, s, field, tab, g, iso, first, tile, cap, cubes, hs.keys,
               slots - 1, hs.vslot, hs.ulist, hs.ucount, xyz);
  chain_launch(k_surf_vnormals, blocks_for(8ll * verts, 128), 128, 0, s, field, g, iso, hs.keys, hs.ulist, hs.ucount,
               hs.nslot, b.pos[cur], b.cell_start, b.scenes, P);
  chain_launch(k_surf_normals, blocks_for(verts, 256), 256, 0, s, hs.vslot, hs.nslot, nrm, verts);
  return cudaGetLastError();
}

}  // namespace pbf
