// PBF step kernels for sm_103a (FP32 on CUDA cores; the step is a sparse
// stencil with no dense contraction, so no tensor cores).
//
// One step (Particles::timeStep, particles.cpp:250-297) is this launch chain
// on one stream; every phase covers all scenes of a batch in one launch (a small
// scene's step is one launch instead, pbf_small.cu):
//   k_predict     gravity + predicted move + collision, cell key, per-cell
//                 count and rank (particles.cpp:175-183, 87-132)
//   k_scan_*      exclusive prefix sum of the cell counts
//   k_scatter     slot = cell start + rank (atomic order within a cell)
//   k_cellrank    order each cell's slots by x, then original index (determinism)
//   k_gather      reorder x, delta, id into cell order; x* = x + delta
//   k_nbr_build   neighbour sets |x*_i - x*_j|^2 <= H2 over the 27 cells,
//                 stored row-compressed (particles.cpp:258-265)
//   k_lambda      density + lambda            (particles.cpp:185-204)   x iters
//   k_deltap      delta p + collision         (particles.cpp:206-213)   x iters
//   k_xsph        velocity, vorticity, XSPH, reported density
//                 (particles.cpp:215-234, order-independent form)
//   k_vort        vorticity confinement, x <- x* (particles.cpp:236-248)
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "pbf_device.cuh"
#include "pbf_nbr.cuh"
#include "pbf_step.cuh"

namespace pbf {
namespace {

constexpr int kScanItems = 4;
constexpr int kScanThreads = 256;
constexpr int kScanTile = kScanItems * kScanThreads;
constexpr uint32_t kSmallCell = 32;       // cells up to this size: ranked slot by slot (k_cellrank)
constexpr uint32_t kMaxSortedCell = 4096;  // larger cells: rank sort by one block (in shared memory)
constexpr int kBigSortThreads = 256;
constexpr int kBigSortBlocks = 64;

// ---------------------------------------------------------------------------
// prediction + cell count
// ---------------------------------------------------------------------------
// REC (recording forward of the adjoint) also stores the collision record in disp.w.
template <bool REC>
__global__ void k_predict(const float4* __restrict__ pos, const float4* __restrict__ vel,
                          float4* __restrict__ disp_out, uint32_t* __restrict__ key_out,
                          uint32_t* __restrict__ xkey_out, uint32_t* __restrict__ rank_out,
                          uint32_t* __restrict__ cell_count,
                          const SceneDesc* __restrict__ scenes, DevParams P, float dt, int move,
                          int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  uint32_t key = 0xffffffffu;
  if (live) {
    const float4 x4 = pos[i];
    const SceneDesc& sc = scenes[scene_of_slot(x4)];
    const float3 x = f3(x4);
    float3 d = make_float3(0.f, 0.f, 0.f);
    if (move) {
      const float4 v4 = vel[i];
      uint32_t code = 0u;
      collide<REC>(x, d, predict_delta(v4, P, dt), true, sc, P, &code);
      disp_out[i] = make_float4(d.x, d.y, d.z, REC ? __uint_as_float(code) : 0.f);
    }
    const float3 xp = displaced(x, d);  // x*, as k_gather forms it
    key = cell_key(cell_of(xp, sc, P.inv_cell), sc);
    key_out[i] = key;
    xkey_out[i] = order_bits(xp.x);
  }
  const uint32_t rank = count_rank(key, live, cell_count);
  if (live) rank_out[i] = rank;
}

// ---------------------------------------------------------------------------
// exclusive scan of cell counts (three phases)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= static_cast<unsigned>(o)) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t w = lane < static_cast<unsigned>(nw) ? warp_sums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= static_cast<unsigned>(o)) w += y;
    }
    if (lane < static_cast<unsigned>(nw)) warp_sums[lane] = w;
  }
  __syncthreads();
  const uint32_t warp_off = warp ? warp_sums[warp - 1] : 0u;
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_off + x - v;
}

// Exclusive scan of the tile sums in place (carry over rounds of blockDim.x); start[m] =
// the total. zero_word (or null): a counter the following phases need at zero (the cell
// sort's worklist). The sums are read through L2: they may come from other blocks.
__device__ __forceinline__ void scan_tile_sums(uint32_t* __restrict__ tile_sum, uint32_t tiles,
                                               uint32_t* __restrict__ start, uint32_t m,
                                               uint32_t* __restrict__ zero_word) {
  if (zero_word && threadIdx.x == 0) *zero_word = 0u;
  uint32_t carry = 0;
  for (uint32_t b = 0; b < tiles; b += blockDim.x) {
    const uint32_t idx = b + threadIdx.x;
    const uint32_t v = idx < tiles ? __ldcg(&tile_sum[idx]) : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, &total);
    if (idx < tiles) tile_sum[idx] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) start[m] = carry;
}

// Scan of each tile of kScanTile counts. CLEAR: the counts are left at zero, as the next step's
// counting expects them. With a ticket (a zeroed word), the last block to
// finish also scans the tile sums (no block waits: each block counts itself in after its
// sum is visible, and the one that counts last does the work, then clears the ticket).
template <bool CLEAR>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(uint32_t* __restrict__ count,
                                                              uint32_t* __restrict__ start,
                                                              uint32_t* __restrict__ tile_sum,
                                                              uint32_t m, uint32_t* __restrict__ ticket,
                                                              uint32_t* __restrict__ zero_word) {
  chain_begin();
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < m) ? count[base + k] : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t off = block_exclusive_scan(s, &total);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (CLEAR && base + k < m) count[base + k] = 0u;
    if (base + k < m) start[base + k] = off;
    off += v[k];
  }
  if (!ticket) {
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
    return;
  }
  __shared__ bool last;
  if (threadIdx.x == 0) {
    tile_sum[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (last) {
    scan_tile_sums(tile_sum, gridDim.x, start, m, zero_word);
    if (threadIdx.x == 0) *ticket = 0u;
  }
}

__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* __restrict__ tile_sum, uint32_t tiles,
                                                     uint32_t* __restrict__ start, uint32_t m,
                                                     uint32_t* __restrict__ zero_word) {
  chain_begin();
  scan_tile_sums(tile_sum, tiles, start, m, zero_word);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_add(uint32_t* __restrict__ start,
                                                            const uint32_t* __restrict__ tile_sum,
                                                            uint32_t m) {
  chain_begin();
  const uint32_t add = tile_sum[blockIdx.x];
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < m) start[base + k] += add;
}

// ---------------------------------------------------------------------------
// reorder
// ---------------------------------------------------------------------------
__global__ void k_scatter(const uint32_t* __restrict__ key, const uint32_t* __restrict__ rank,
                          const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ perm, int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) perm[cell_start[key[i]] + rank[i]] = static_cast<uint32_t>(i);
}

// Order each cell's slots by the x coordinate of x* (pos + disp, as k_gather forms it;
// pos for a resort), ties by original particle index: the cell order (hence every
// neighbour sum) is independent of atomic timing, and since cells along x are adjacent
// slot ranges, every row of cells is sorted by x, which lets the neighbour build stop a
// row at the first candidate beyond the reach. Cells up to kSmallCell particles are
// ranked by k_cellrank; larger ones go to a worklist for k_cellsort_big.
// The x keys (order_bits of x*.x) are written by k_predict, indexed by the pre-sort slot.
__device__ __forceinline__ uint64_t slot_order_key(const uint32_t* __restrict__ xkey, const uint32_t* __restrict__ id,
                                                   uint32_t v) {
  return (static_cast<uint64_t>(xkey[v]) << 32) | id[v];
}

// One thread per slot s of the scatter's (atomic) order: the entry moves to its cell's
// start plus its rank, the number of the cell's entries with a smaller key (keys are
// distinct). A cell's threads are neighbours, so its keys are read from L1. Cells over
// kSmallCell particles are copied in atomic order and listed for k_cellsort_big (their
// first slot's thread adds them).
__global__ void k_cellrank(const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ atomic_order,
                           const uint32_t* __restrict__ key, const uint32_t* __restrict__ xkey,
                           const uint32_t* __restrict__ id, uint32_t* __restrict__ perm,
                           uint32_t* __restrict__ big_cells, uint32_t* __restrict__ big_count, int n) {
  chain_begin();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint32_t v = atomic_order[s];
  const uint32_t c = key[v];
  const uint32_t b = cell_start[c], e = cell_start[c + 1];
  if (e - b > kSmallCell) {
    perm[s] = v;
    if (static_cast<uint32_t>(s) == b) big_cells[atomicAdd(big_count, 1u)] = c;
    return;
  }
  const uint64_t kv = slot_order_key(xkey, id, v);
  uint32_t r = 0;
  for (uint32_t u = b; u < e; ++u) r += slot_order_key(xkey, id, atomic_order[u]) < kv ? 1u : 0u;
  perm[b + r] = v;
}

// Rank sort of the worklist's cells, one block per cell: the rank of an element is the
// number of the cell's elements with a smaller key (keys are distinct). Cells over
// kMaxSortedCell particles keep the atomic order (bounded time); such a cell makes its
// rows exceed kMaxRowCandidates, which the neighbour build reports as an error.
__global__ void __launch_bounds__(kBigSortThreads) k_cellsort_big(const uint32_t* __restrict__ cell_start,
                                                                 uint32_t* __restrict__ perm,
                                                                 const uint32_t* __restrict__ xkey,
                                                                 const uint32_t* __restrict__ id,
                                                                 const uint32_t* __restrict__ big_cells,
                                                                 const uint32_t* __restrict__ big_count) {
  chain_begin();
  __shared__ uint32_t slot[kMaxSortedCell];
  __shared__ uint32_t khi[kMaxSortedCell];
  __shared__ uint32_t klo[kMaxSortedCell];
  const uint32_t cnt = *big_count;
  for (uint32_t w = blockIdx.x; w < cnt; w += gridDim.x) {
    const uint32_t c = big_cells[w];
    const uint32_t b = cell_start[c], e = cell_start[c + 1];
    const uint32_t m = e - b;
    if (m > kMaxSortedCell) continue;  // uniform across the block
    for (uint32_t t = threadIdx.x; t < m; t += blockDim.x) {
      const uint32_t v = perm[b + t];
      const uint64_t k = slot_order_key(xkey, id, v);
      slot[t] = v;
      khi[t] = static_cast<uint32_t>(k >> 32);
      klo[t] = static_cast<uint32_t>(k);
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < m; t += blockDim.x) {
      const uint32_t kh = khi[t], kl = klo[t];
      uint32_t r = 0;
      for (uint32_t u = 0; u < m; ++u) r += (khi[u] < kh || (khi[u] == kh && klo[u] < kl)) ? 1u : 0u;
      perm[b + r] = slot[t];
    }
    __syncthreads();
  }
}

__global__ void k_gather(const uint32_t* __restrict__ perm, const float4* __restrict__ pos_a,
                         const float4* __restrict__ disp_a, const float4* __restrict__ vel_a,
                         const uint32_t* __restrict__ id_a, float4* __restrict__ pos_b,
                         float4* __restrict__ disp_b, float4* __restrict__ xs_b,
                         float4* __restrict__ vel_b, uint32_t* __restrict__ id_b, int n) {
  chain_begin();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint32_t i = perm[s];
  const float4 x = pos_a[i];
  pos_b[s] = x;
  id_b[s] = id_a[i];
  float rec = 0.f;
  if (disp_a) {
    const float4 d = disp_a[i];
    disp_b[s] = d;
    const float3 xs = displaced(f3(x), f3(d));
    xs_b[s] = make_float4(xs.x, xs.y, xs.z, 0.f);
    rec = d.w;
  }
  if (vel_a) {  // with disp_a (recording forward): w carries the prediction's collision record
    float4 v = vel_a[i];
    v.w = rec;
    vel_b[s] = v;
  }
}

// ---------------------------------------------------------------------------
// neighbour sets
// ---------------------------------------------------------------------------
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1152 / BLOCK) k_nbr_build(const float4* __restrict__ xs,
                                                     const float4* __restrict__ pos,
                                                     const uint32_t* __restrict__ cell_start,
                                                     const SceneDesc* __restrict__ scenes,
                                                     uint4* __restrict__ hdr, uint32_t* __restrict__ words,
                                                     unsigned* __restrict__ err, DevParams P, float one, int n) {
  chain_begin();
  extern __shared__ uint4 nbr_smem[];
  nbr_build_warp<true, true>(reinterpret_cast<NbrWarp*>(nbr_smem)[threadIdx.x >> 5],
                       static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x), xs, pos, cell_start, scenes, hdr,
                       words, err, P, one, n);
}

// ---------------------------------------------------------------------------
// Jacobi density-constraint iterations
// ---------------------------------------------------------------------------
// lambda_i is stored in x*_i.w of the same buffer: within this pass every
// thread reads only .xyz of its neighbours' x*, which no thread writes.
template <int BLOCK, int D, bool ST>
__global__ void __launch_bounds__(BLOCK) k_lambda(float4* xs, const uint4* __restrict__ hdr,
                                                  const uint32_t* __restrict__ words,
                                                  float* __restrict__ rho_iter0,
                                                  DevParams P, int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = xs[i];
  LambdaSum sum;
  // D gathers in flight
  for_each_neighbor_pf<D, ST>(i, n, ld_hdr<ST>(&hdr[i]), words,
                                              [&](uint32_t j) -> float4 { return xs[j]; },
                                              [&](uint32_t, const float4& xj) { sum.add(xi, xj, P); });
  float rho;
  const float l = sum.lambda(P, &rho);
  reinterpret_cast<float*>(xs)[4 * i + 3] = l;
  if (rho_iter0) rho_iter0[i] = rho;
}

// (lambda_i + lambda_j + s_corr) grad W summed over neighbours; N4 specialises the
// tensile exponent N = 4 of particles.cpp:40. REC (recording forward of the adjoint)
// also stores the requested displacement and the collision record in dp_rec. MESH =
// false (no collider triangles) leaves the triangle tests out of the collision: 40
// registers a thread instead of 55.
template <int BLOCK, bool N4, bool REC, bool MESH, int D, bool ST>
__global__ void __launch_bounds__(BLOCK) k_deltap(const float4* __restrict__ xs,
                                                  const float4* __restrict__ pos,
                                                  const uint4* __restrict__ hdr,
                                                  const uint32_t* __restrict__ words,
                                                  const SceneDesc* __restrict__ scenes,
                                                  float4* __restrict__ disp, float4* __restrict__ xs_next,
                                                  float4* __restrict__ dp_rec, DevParams P, int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = xs[i];
  const float wt = P.poly6_c * P.tis;
  DeltaSum<N4> sum;  // lambda_i is x*_i.w
  for_each_neighbor_pf<D, ST>(i, n, ld_hdr<ST>(&hdr[i]), words,
                                              [&](uint32_t j) -> float4 { return __ldg(&xs[j]); },
                                              [&](uint32_t, const float4& xj) { sum.add(xi, xj, wt, P); });
  const float3 dp = sum.delta(P);
  const float4 x4 = pos[i];
  const SceneDesc& sc = scenes[scene_of_slot(x4)];
  const float4 d4 = disp[i];
  float3 d = f3(d4);
  const float3 x = f3(x4);
  uint32_t code = 0u;
  collide<REC, MESH>(x, d, dp, false, sc, P, &code);
  if (REC) dp_rec[i] = make_float4(dp.x, dp.y, dp.z, __uint_as_float(code));
  disp[i] = make_float4(d.x, d.y, d.z, 0.f);
  const float3 xn = displaced(x, d);
  xs_next[i] = make_float4(xn.x, xn.y, xn.z, 0.f);
}

// ---------------------------------------------------------------------------
// velocity, vorticity, XSPH, reported density; then vorticity confinement
// ---------------------------------------------------------------------------
// |omega_i| is stored in x*_i.w of the same buffer (neighbours read only .xyz here).
template <int BLOCK, int D, bool ST>
__global__ void __launch_bounds__(BLOCK) k_xsph(float4* xs, const float4* __restrict__ disp,
                                                const uint4* __restrict__ hdr,
                                                const uint32_t* __restrict__ words,
                                                float4* __restrict__ vel_out, float4* __restrict__ omega,
                                                float* __restrict__ rho_out, DevParams P, float inv_dt,
                                                int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = xs[i];
  const float3 vi = f3(disp[i]) * inv_dt;  // updateVelocity, particles.cpp:215-217
  XsphSum sum;
  for_each_neighbor_pf<D, ST>(
      i, n, ld_hdr<ST>(&hdr[i]), words, [&](uint32_t j) { return XD{xs[j], __ldg(&disp[j])}; },
      [&](uint32_t, const XD& a) { sum.add(xi, vi, a, inv_dt, P); });
  const float3 v = sum.velocity(vi, P);
  vel_out[i] = make_float4(v.x, v.y, v.z, 0.f);
  const float4 w = sum.omega(P);
  omega[i] = w;
  reinterpret_cast<float*>(xs)[4 * i + 3] = w.w;
  rho_out[i] = sum.rho(P);
}

template <int BLOCK, int D, bool ST>
__global__ void __launch_bounds__(BLOCK) k_vort(const float4* __restrict__ xs,
                                                float4* __restrict__ pos,
                                                const float4* __restrict__ omega,
                                                const uint4* __restrict__ hdr,
                                                const uint32_t* __restrict__ words,
                                                float4* __restrict__ vel, unsigned* __restrict__ err,
                                                float4* __restrict__ eta_rec, DevParams P, float dt, int n) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = xs[i];
  VortSum sum;  // |omega_j| is x*_j.w
  for_each_neighbor_pf<D, ST>(i, n, ld_hdr<ST>(&hdr[i]), words,
                                              [&](uint32_t j) -> float4 { return __ldg(&xs[j]); },
                                              [&](uint32_t, const float4& xj) { sum.add(xi, xj, P); });
  const float3 eta = sum.location(P);
  if (eta_rec) eta_rec[i] = make_float4(eta.x, eta.y, eta.z, 0.f);  // recording forward of the adjoint
  const float3 v = confined(f3(vel[i]), eta, omega[i], dt, P);
  const float4 p4 = pos[i];
  vel[i] = make_float4(v.x, v.y, v.z, 0.f);
  pos[i] = make_float4(xi.x, xi.y, xi.z, p4.w);  // updatePosition, particles.cpp:246-248
  if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(xi.x) && isfinite(xi.y) &&
        isfinite(xi.z)))
    atomicOr(err, PBF_ERRBIT_NONFINITE);
}

// Step statistics (the prints of particles.cpp:267-295 and the neighbour
// alert of :168-172, as numbers): one pass over densities and list headers, reduced in
// a fixed shape (kStatsBlocks partial records, then one block), so the sums are
// deterministic and no block contends on an atomic.

__device__ __forceinline__ void stats_merge(DevStats& a, const DevStats& b) {
  a.rho_sum += b.rho_sum;
  a.rho_iter0_sum += b.rho_iter0_sum;
  a.err_sum += b.err_sum;
  a.err_max_bits = max(a.err_max_bits, b.err_max_bits);  // non-negative floats order as their bits
  a.nbr_min = min(a.nbr_min, b.nbr_min);
  a.nbr_max = max(a.nbr_max, b.nbr_max);
  a.nbr_sum += b.nbr_sum;
  a.low_cnt += b.low_cnt;
}

__device__ __forceinline__ DevStats stats_shfl_down(const DevStats& a, int o) {
  DevStats b;
  b.rho_sum = __shfl_down_sync(0xffffffffu, a.rho_sum, o);
  b.rho_iter0_sum = __shfl_down_sync(0xffffffffu, a.rho_iter0_sum, o);
  b.err_sum = __shfl_down_sync(0xffffffffu, a.err_sum, o);
  b.err_max_bits = __shfl_down_sync(0xffffffffu, a.err_max_bits, o);
  b.nbr_min = __shfl_down_sync(0xffffffffu, a.nbr_min, o);
  b.nbr_max = __shfl_down_sync(0xffffffffu, a.nbr_max, o);
  b.nbr_sum = __shfl_down_sync(0xffffffffu, a.nbr_sum, o);
  b.low_cnt = __shfl_down_sync(0xffffffffu, a.low_cnt, o);
  return b;
}

// Reduces the block's records into thread 0 (blockDim.x a multiple of 32, at most 1024).
__device__ __forceinline__ DevStats stats_block_reduce(DevStats a) {
  __shared__ DevStats sw[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) stats_merge(a, stats_shfl_down(a, o));
  const unsigned w = threadIdx.x >> 5;
  if (lane_id() == 0) sw[w] = a;
  __syncthreads();
  if (threadIdx.x == 0)
    for (unsigned k = 1; k < (blockDim.x >> 5); ++k) stats_merge(a, sw[k]);
  return a;
}

__device__ __forceinline__ DevStats stats_zero() {
  DevStats a;
  a.rho_sum = a.rho_iter0_sum = a.err_sum = 0.0;
  a.err_max_bits = 0u;
  a.nbr_min = 0xffffffffu;
  a.nbr_max = 0u;
  a.pad = 0u;
  a.nbr_sum = a.low_cnt = 0ull;
  return a;
}

// Each thread takes 4 consecutive particles per turn (vector loads of the densities, the
// 4 list headers issued together) and sums its share (about 16 particles at 1M) in FP32;
// the partial sums join in FP64 from the warp level up. FP64 adds per particle would
// bound the kernel: FP64 throughput on this part is a small fraction of FP32's.
struct StatsAcc {
  float rho, rho0, err, err_max;
  unsigned nmin, nmax, nsum, low;
};

__device__ __forceinline__ void stats_add(StatsAcc& a, float x, float x0, unsigned c, float inv_rho0) {
  a.rho += x;
  a.rho0 += x0;
  const float e = fabsf(x * inv_rho0 - 1.0f);
  a.err += e;
  a.err_max = fmaxf(a.err_max, e);
  a.nmin = min(a.nmin, c);
  a.nmax = max(a.nmax, c);
  a.nsum += c;
  a.low += c < static_cast<unsigned>(kNeighborAlert) ? 1u : 0u;
}

// JOIN: the last block to finish joins the partial records itself (its threads take one each), which
// saves a small scene's step the launch of k_stats_final.
static_assert(kStatsBlocks == 256, "a block's threads take one partial record each");
template <bool JOIN>
__global__ void __launch_bounds__(256) k_stats(const float* __restrict__ rho, const float* __restrict__ rho0,
                                               const uint4* __restrict__ hdr, DevStats* part,
                                               DevStats* __restrict__ st, unsigned* ticket, float inv_rho0, int n) {
  chain_begin();
  StatsAcc s{0.f, 0.f, 0.f, 0.f, 0xffffffffu, 0u, 0u, 0u};
  const int n4 = n / 4;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n4; k += gridDim.x * blockDim.x) {
    const float4 x = reinterpret_cast<const float4*>(rho)[k];
    const float4 x0 = reinterpret_cast<const float4*>(rho0)[k];
    const uint4 h0 = hdr[4 * k], h1 = hdr[4 * k + 1], h2 = hdr[4 * k + 2], h3 = hdr[4 * k + 3];
    stats_add(s, x.x, x0.x, h0.w, inv_rho0);
    stats_add(s, x.y, x0.y, h1.w, inv_rho0);
    stats_add(s, x.z, x0.z, h2.w, inv_rho0);
    stats_add(s, x.w, x0.w, h3.w, inv_rho0);
  }
  const int t = 4 * n4 + blockIdx.x * blockDim.x + threadIdx.x;  // the last n % 4 particles
  if (t < n) stats_add(s, rho[t], rho0[t], static_cast<unsigned>(nbr_total(hdr[t])), inv_rho0);
  DevStats a = stats_zero();
  a.rho_sum = s.rho;
  a.rho_iter0_sum = s.rho0;
  a.err_sum = s.err;
  a.err_max_bits = __float_as_uint(s.err_max);
  a.nbr_min = s.nmin;
  a.nbr_max = s.nmax;
  a.nbr_sum = s.nsum;
  a.low_cnt = s.low;
  a = stats_block_reduce(a);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a;
    if (JOIN) {  // counted in last: the ticket wraps to zero
      __threadfence();
      last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
      __threadfence();
    }
  }
  if (!JOIN) return;
  __syncthreads();
  if (!last) return;
  static_assert(sizeof(DevStats) % 8 == 0, "read as 8-byte words");
  unsigned long long w[sizeof(DevStats) / 8];
#pragma unroll
  for (size_t k = 0; k < sizeof(DevStats) / 8; ++k)
    w[k] = __ldcg(reinterpret_cast<const unsigned long long*>(&part[threadIdx.x]) + k);
  memcpy(&a, w, sizeof(a));
  a = stats_block_reduce(a);
  if (threadIdx.x == 0) *st = a;
}

__global__ void __launch_bounds__(kStatsBlocks) k_stats_final(const DevStats* __restrict__ part,
                                                              DevStats* __restrict__ st) {
  chain_begin();
  DevStats a = part[threadIdx.x];
  a = stats_block_reduce(a);
  if (threadIdx.x == 0) *st = a;
}

// ---------------------------------------------------------------------------
// transfers between original order and cell order
// ---------------------------------------------------------------------------
__global__ void k_upload(const float* __restrict__ xyz, const float* __restrict__ v,
                         const SceneDesc* __restrict__ scenes, int n_scenes, float4* __restrict__ pos,
                         float4* __restrict__ vel, uint32_t* __restrict__ id, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int lo = 0, hi = n_scenes - 1;  // scene whose particle range holds s
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (scenes[mid].p_off <= static_cast<uint32_t>(s)) lo = mid; else hi = mid - 1;
  }
  pos[s] = make_float4(xyz[3 * s], xyz[3 * s + 1], xyz[3 * s + 2], __int_as_float(lo));
  vel[s] = v ? make_float4(v[3 * s], v[3 * s + 1], v[3 * s + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
  id[s] = static_cast<uint32_t>(s);
}

__global__ void k_download(const float4* __restrict__ pos, const float4* __restrict__ vel,
                           const float* __restrict__ rho, const uint32_t* __restrict__ id,
                           float* __restrict__ xyz, float* __restrict__ v, float* __restrict__ r, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint32_t o = id[s];
  if (xyz) {
    const float4 p = pos[s];
    xyz[3 * o] = p.x;
    xyz[3 * o + 1] = p.y;
    xyz[3 * o + 2] = p.z;
  }
  if (v) {
    const float4 q = vel[s];
    v[3 * o] = q.x;
    v[3 * o + 1] = q.y;
    v[3 * o + 2] = q.z;
  }
  if (r) r[o] = rho[s];
}

__global__ void k_unsort_u32(const uint32_t* __restrict__ src, const uint32_t* __restrict__ id,
                             uint32_t* __restrict__ dst, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) dst[id[s]] = src[s];
}

__global__ void k_unsort_f4(const float4* __restrict__ src, const uint32_t* __restrict__ id,
                            float* __restrict__ dst, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float4 p = src[s];
  const uint32_t o = id[s];
  dst[3 * o] = p.x;
  dst[3 * o + 1] = p.y;
  dst[3 * o + 2] = p.z;
}

__global__ void k_cells_of(const float4* __restrict__ xs, const float4* __restrict__ pos,
                           const SceneDesc* __restrict__ scenes, const uint32_t* __restrict__ id,
                           uint32_t* __restrict__ cells, DevParams P, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const SceneDesc& sc = scenes[scene_of_slot(pos[s])];
  cells[id[s]] = cell_key(cell_of(f3(xs[s]), sc, P.inv_cell), sc);
}

__global__ void k_nbr_counts(const uint4* __restrict__ hdr, const uint32_t* __restrict__ id,
                             uint32_t* __restrict__ counts, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) counts[id[s]] = static_cast<uint32_t>(nbr_total(hdr[s]));
}

// ids[offsets[id[i]] ...] = original ids of i's neighbours (cell order).
__global__ void k_nbr_ids(const uint4* __restrict__ hdr, const uint32_t* __restrict__ words,
                          const uint32_t* __restrict__ id, const uint32_t* __restrict__ offsets,
                          uint32_t* __restrict__ ids, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t o = offsets[id[i]];
  for_each_neighbor(i, n, hdr[i], words, [&](uint32_t j) { ids[o++] = id[j]; });
}

// Particles::estimateDensities (particles.cpp:440-444) on cell-sorted x: self included.
__global__ void k_density_self(const float4* __restrict__ pos, const uint32_t* __restrict__ cell_start,
                               const SceneDesc* __restrict__ scenes, float* __restrict__ rho,
                               DevParams P, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = pos[i];
  const SceneDesc& sc = scenes[scene_of_slot(xi)];
  const CellCoord cc = cell_of(f3(xi), sc, P.inv_cell);
  float qsum = 0.f;
  for (int r = 0; r < 9; ++r) {
    const int z = cc.z + r / 3 - 1, y = cc.y + r % 3 - 1;
    if (z < 0 || z >= sc.dim[2] || y < 0 || y >= sc.dim[1]) continue;
    const uint32_t row = sc.cell_off + static_cast<uint32_t>((z * sc.dim[1] + y) * sc.dim[0]);
    const int x0 = cc.x > 0 ? cc.x - 1 : 0;
    const int x1 = cc.x + 1 < sc.dim[0] ? cc.x + 1 : sc.dim[0] - 1;
    for (uint32_t j = cell_start[row + x0]; j < cell_start[row + x1 + 1]; ++j) {
      const float4 xj = __ldg(&pos[j]);
      const float3 d = make_float3(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z);
      const float r2 = dot3(d, d);
      if (r2 < P.h2) {
        const float q = P.h2 - r2;
        qsum += q * q * q;
      }
    }
  }
  rho[i] = P.poly6_c * qsum;
}

// Particles::estimateDensityAt (particles.cpp:446-453) at query points, scene 0.
__global__ void k_density_at(const float4* __restrict__ pos, const uint32_t* __restrict__ cell_start,
                             const SceneDesc* __restrict__ scenes, const float* __restrict__ pts,
                             float* __restrict__ out, DevParams P, int m) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  out[q] = density_at_point(make_float3(pts[3 * q], pts[3 * q + 1], pts[3 * q + 2]), pos, cell_start, scenes[0], P);
}

inline unsigned blocks_for(size_t n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

// Launches neighbour kernel KERN (a template-id, parenthesised) over n particles, BLOCK threads a block.
#define PBF_PASS_LAUNCH(KERN, ...) chain_launch(KERN, blocks_for(n, BLOCK), BLOCK, 0, s, __VA_ARGS__)

// Instantiates a neighbour pass for the tuned gather depth (D = 4 or 8 neighbour loads in
// flight per thread) and list-load policy (ST: streaming). Neither changes the order in
// which a particle's neighbours are summed, so every form gives the same bits.
#define PBF_FORM_SWITCH(depth, stream, ...)                                          \
  if ((depth) == 4) {                                                                \
    if (stream) { constexpr int D = 4; constexpr bool ST = true; __VA_ARGS__; }      \
    else { constexpr int D = 4; constexpr bool ST = false; __VA_ARGS__; }            \
  } else {                                                                           \
    if (stream) { constexpr int D = 8; constexpr bool ST = true; __VA_ARGS__; }      \
    else { constexpr int D = 8; constexpr bool ST = false; __VA_ARGS__; }            \
  }

// The neighbour build; blocks of 256 and 512 threads need more shared memory than a kernel has by default.
template <int BLOCK>
cudaError_t launch_nbr_build(const Buffers& b, const DevParams& P, const float4* xs, const float4* pos,
                             cudaStream_t s) {
  constexpr size_t bytes = sizeof(NbrWarp) * (BLOCK / 32);
  const int n = static_cast<int>(b.n);
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_nbr_build<BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
  }
  chain_launch(k_nbr_build<BLOCK>, blocks_for(n, BLOCK), BLOCK, bytes, s, xs, pos, b.cell_start, b.scenes, b.nbr_hdr,
               b.nbr_w, b.err, P, 1.0f, n);
  return cudaGetLastError();
}

void launch_stats(const Buffers& b, const DevParams& P, bool join, cudaStream_t s) {
  auto kern = join ? k_stats<true> : k_stats<false>;
  chain_launch(kern, kStatsBlocks, 256, 0, s, b.rho, b.rho_iter0, b.nbr_hdr, b.stats_part, b.stats, b.grid_bar + 2,
               P.inv_rho0, static_cast<int>(b.n));
  if (!join) chain_launch(k_stats_final, 1, kStatsBlocks, 0, s, b.stats_part, b.stats);
}

// One delta-p pass (B = the buffer index holding this step's cell-ordered x and delta).
// The recording forward of the adjoint keeps the default form (8 deep, cached lists).
template <bool N4, bool REC, bool MESH>
void launch_deltap(const Tuning& t, const Buffers& b, int B, float4* xcur, float4* xnext, float4* dprec,
                   const DevParams& P, int n, cudaStream_t s) {
  if (REC) {
    PBF_BLOCK_SWITCH(t.block_solve,
                     PBF_PASS_LAUNCH((k_deltap<BLOCK, N4, REC, MESH, 8, false>), xcur, b.pos[B], b.nbr_hdr,
                                     b.nbr_w, b.scenes, b.disp[1], xnext, dprec, P, n));
    return;
  }
  PBF_FORM_SWITCH(t.gather_depth, t.list_stream,
                  PBF_BLOCK_SWITCH(t.block_solve,
                                   PBF_PASS_LAUNCH((k_deltap<BLOCK, N4, REC, MESH, D, ST>), xcur, b.pos[B],
                                                   b.nbr_hdr, b.nbr_w, b.scenes, b.disp[1], xnext, dprec, P, n)));
}

// Shared front half of a step and of a resort: keys, counts, scan, slots. Its first kernel is launched
// plainly: what comes before it in the stream may be a wait for another stream's event.
cudaError_t sort_into_cells(const Buffers& b, const DevParams& P, const Tuning& t, int cur, float dt,
                            bool move, cudaStream_t s, PhaseMarks* mk = nullptr, bool rec = false) {
  const int n = static_cast<int>(b.n);
  const uint32_t m = b.n_cells;
  if (rec)
    k_predict<true><<<blocks_for(n, t.block_predict), t.block_predict, 0, s>>>(
        b.pos[cur], b.vel[cur], b.disp[0], b.key, b.xkey, b.rank, b.cell_count, b.scenes, P, dt, move ? 1 : 0, n);
  else
    k_predict<false><<<blocks_for(n, t.block_predict), t.block_predict, 0, s>>>(
        b.pos[cur], b.vel[cur], b.disp[0], b.key, b.xkey, b.rank, b.cell_count, b.scenes, P, dt, move ? 1 : 0, n);
  if (mk) mk->mark(kPhasePredict, s);
  const uint32_t tiles = (m + kScanTile - 1) / kScanTile;
  // scan_tmp holds the tile sums and, after them, the ticket of k_scan_tiles' last block
  chain_launch(k_scan_tiles<true>, tiles, kScanThreads, 0, s, b.cell_count, b.cell_start, b.scan_tmp, m,
               b.scan_tmp + tiles, b.big_count);
  chain_launch(k_scan_add, tiles, kScanThreads, 0, s, b.cell_start, b.scan_tmp, m);
  if (mk) mk->mark(kPhaseScan, s);
  chain_launch(k_scatter, blocks_for(n, t.block_misc), t.block_misc, 0, s, b.key, b.rank, b.cell_start, b.perm_atomic,
               n);
  chain_launch(k_cellrank, blocks_for(n, t.block_misc), t.block_misc, 0, s, b.cell_start, b.perm_atomic, b.key, b.xkey,
               b.id[cur], b.perm, b.big_cells, b.big_count, n);
  chain_launch(k_cellsort_big, kBigSortBlocks, kBigSortThreads, 0, s, b.cell_start, b.perm, b.xkey, b.id[cur],
               b.big_cells, b.big_count);
  if (mk) mk->mark(kPhaseSort, s);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_step(const Buffers& b, const DevParams& P, const Tuning& t, int cur, float dt,
                        int iters, bool keep_pred, cudaStream_t s, PhaseMarks* mk, const Tape* tape) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  const int A = cur, B = 1 - cur;
  const bool rec = tape != nullptr;
  const int form = !rec && !mk ? small_step_form(b, P) : 0;
  if (form) {
    cudaError_t es = launch_step_small(b, P, form, cur, dt, iters, keep_pred, s);
    if (es != cudaSuccess) return es;
    if (P.stats) launch_stats(b, P, true, s);
    return cudaGetLastError();
  }
  if (mk) mk->mark(-1, s);
  cudaError_t e = sort_into_cells(b, P, t, A, dt, true, s, mk, rec);
  if (e != cudaSuccess) return e;
  float4* xs0 = rec ? tape->xs : b.xs[0];
  chain_launch(k_gather, blocks_for(n, t.block_misc), t.block_misc, 0, s, b.perm, b.pos[A], b.disp[0],
               rec ? b.vel[A] : nullptr, b.id[A], b.pos[B], b.disp[1], xs0, rec ? tape->v : nullptr, b.id[B], n);
  if (rec) {
    e = cudaMemcpyAsync(tape->x, b.pos[B], sizeof(float4) * b.n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  if (keep_pred && b.pred) {
    e = cudaMemcpyAsync(b.pred, xs0, sizeof(float4) * b.n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  if (mk) mk->mark(kPhaseGather, s);
  PBF_BLOCK_SWITCH(t.block_nbr, e = launch_nbr_build<BLOCK>(b, P, xs0, b.pos[B], s));
  if (e != cudaSuccess) return e;
  if (mk) mk->mark(kPhaseNeighbors, s);
  for (int it = 0; it < iters; ++it) {
    float4* xcur = rec ? tape->xs + static_cast<size_t>(it) * b.n : b.xs[it & 1];
    float4* xnext = rec ? tape->xs + static_cast<size_t>(it + 1) * b.n : b.xs[(it + 1) & 1];
    float4* dprec = rec ? tape->dp + static_cast<size_t>(it) * b.n : nullptr;
    PBF_FORM_SWITCH(t.gather_depth, t.list_stream,
                    PBF_BLOCK_SWITCH(t.block_solve,
                                     PBF_PASS_LAUNCH((k_lambda<BLOCK, D, ST>), xcur, b.nbr_hdr,
                                                     b.nbr_w, (it == 0 && P.stats) ? b.rho_iter0 : nullptr, P,
                                                     n)));
    if (mk) mk->mark(kPhaseLambda, s);
    const bool n4 = P.scorr_n == 4, mesh = P.n_mesh > 0 || P.n_sph > 0;
    if (rec) {  // the adjoint takes box colliders only; the recording keeps the general form
      if (n4) launch_deltap<true, true, true>(t, b, B, xcur, xnext, dprec, P, n, s);
      else launch_deltap<false, true, true>(t, b, B, xcur, xnext, dprec, P, n, s);
    } else if (n4) {
      if (mesh) launch_deltap<true, false, true>(t, b, B, xcur, xnext, nullptr, P, n, s);
      else launch_deltap<true, false, false>(t, b, B, xcur, xnext, nullptr, P, n, s);
    } else {
      if (mesh) launch_deltap<false, false, true>(t, b, B, xcur, xnext, nullptr, P, n, s);
      else launch_deltap<false, false, false>(t, b, B, xcur, xnext, nullptr, P, n, s);
    }
    if (mk) mk->mark(kPhaseDeltaP, s);
  }
  float4* fin = rec ? tape->xs + static_cast<size_t>(iters) * b.n : b.xs[iters & 1];
  PBF_FORM_SWITCH(t.gather_depth, t.list_stream,
                  PBF_BLOCK_SWITCH(t.block_solve,
                                   PBF_PASS_LAUNCH((k_xsph<BLOCK, D, ST>), fin, b.disp[1],
                                                   b.nbr_hdr, b.nbr_w, b.vel[B], b.omega, b.rho, P, 1.0f / dt, n)));
  if (mk) mk->mark(kPhaseXsph, s);
  PBF_FORM_SWITCH(t.gather_depth, t.list_stream,
                  PBF_BLOCK_SWITCH(t.block_solve,
                                   PBF_PASS_LAUNCH((k_vort<BLOCK, D, ST>), fin, b.pos[B], b.omega,
                                                   b.nbr_hdr, b.nbr_w, b.vel[B], b.err, rec ? tape->eta : nullptr,
                                                   P, dt, n)));
  if (mk) mk->mark(kPhaseVorticity, s);
  if (P.stats) {
    launch_stats(b, P, false, s);
  }
  if (mk) mk->mark(kPhaseStats, s);
  return cudaGetLastError();
}

// Reorder the state into cells of the current positions (no motion); the
// result lands in buffers 1 - cur.
cudaError_t launch_resort(const Buffers& b, const DevParams& P, const Tuning& t, int cur, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  cudaError_t e = sort_into_cells(b, P, t, cur, 0.f, false, s);
  if (e != cudaSuccess) return e;
  chain_launch(k_gather, blocks_for(n, t.block_misc), t.block_misc, 0, s, b.perm, b.pos[cur], nullptr, b.vel[cur],
               b.id[cur], b.pos[1 - cur], nullptr, nullptr, b.vel[1 - cur], b.id[1 - cur], n);
  return cudaGetLastError();
}

cudaError_t launch_upload(const Buffers& b, int cur, const float* xyz, const float* vel,
                          const uint32_t* /*scene_of*/, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_upload<<<blocks_for(n, 256), 256, 0, s>>>(xyz, vel, b.scenes, b.n_scenes, b.pos[cur], b.vel[cur],
                                              b.id[cur], n);
  return cudaGetLastError();
}

cudaError_t launch_download(const Buffers& b, int cur, float* xyz, float* vel, float* rho, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_download<<<blocks_for(n, 256), 256, 0, s>>>(b.pos[cur], b.vel[cur], b.rho, b.id[cur], xyz, vel, rho, n);
  return cudaGetLastError();
}

cudaError_t launch_unsort_u32(const Buffers& b, int cur, const uint32_t* src, uint32_t* dst, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_unsort_u32<<<blocks_for(n, 256), 256, 0, s>>>(src, b.id[cur], dst, n);
  return cudaGetLastError();
}

cudaError_t launch_unsort_f4(const Buffers& b, int cur, const float4* src, float* dst_xyz, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_unsort_f4<<<blocks_for(n, 256), 256, 0, s>>>(src, b.id[cur], dst_xyz, n);
  return cudaGetLastError();
}

cudaError_t launch_cells_of(const Buffers& b, const DevParams& P, int cur, uint32_t* cells, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_cells_of<<<blocks_for(n, 256), 256, 0, s>>>(b.pred, b.pos[cur], b.scenes, b.id[cur], cells, P, n);
  return cudaGetLastError();
}

cudaError_t launch_neighbor_counts(const Buffers& b, int cur, uint32_t* counts, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_nbr_counts<<<blocks_for(n, 256), 256, 0, s>>>(b.nbr_hdr, b.id[cur], counts, n);
  return cudaGetLastError();
}

cudaError_t launch_neighbor_ids(const Buffers& b, int cur, const uint32_t* offsets, uint32_t* ids,
                                cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_nbr_ids<<<blocks_for(n, 256), 256, 0, s>>>(b.nbr_hdr, b.nbr_w, b.id[cur], offsets, ids, n);
  return cudaGetLastError();
}

cudaError_t launch_exclusive_scan(const uint32_t* count, uint32_t* start, uint32_t* tile_sums, uint32_t m,
                                  cudaStream_t s) {
  const uint32_t tiles = (m + kScanTile - 1) / kScanTile;
  chain_launch(k_scan_tiles<false>, tiles, kScanThreads, 0, s, const_cast<uint32_t*>(count), start, tile_sums, m,
               nullptr, nullptr);
  chain_launch(k_scan_sums, 1, 1024, 0, s, tile_sums, tiles, start, m, nullptr);
  chain_launch(k_scan_add, tiles, kScanThreads, 0, s, start, tile_sums, m);
  return cudaGetLastError();
}

uint32_t exclusive_scan_tiles(uint32_t m) { return (m + kScanTile - 1) / kScanTile; }

cudaError_t launch_density_self(const Buffers& b, const DevParams& P, const Tuning& t, int cur,
                                float* rho_sorted, cudaStream_t s) {
  const int n = static_cast<int>(b.n);
  if (n == 0) return cudaSuccess;
  k_density_self<<<blocks_for(n, t.block_misc), t.block_misc, 0, s>>>(b.pos[cur], b.cell_start, b.scenes,
                                                                       rho_sorted, P, n);
  return cudaGetLastError();
}

cudaError_t launch_density_at(const Buffers& b, const DevParams& P, int cur, size_t m, const float* pts,
                              float* out, cudaStream_t s) {
  if (m == 0) return cudaSuccess;
  k_density_at<<<blocks_for(m, 256), 256, 0, s>>>(b.pos[cur], b.cell_start, b.scenes, pts, out, P,
                                                  static_cast<int>(m));
  return cudaGetLastError();
}

}  // namespace pbf
