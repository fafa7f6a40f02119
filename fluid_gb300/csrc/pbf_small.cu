// One step of a small scene in one launch: the phases of launch_step (pbf_kernels.cu) as the
// stages of a cooperative kernel, every block resident, and a barrier over the grid between
// stages.
//
// What bounds a small step is not work but latency: about 20 dependent launches, and in each
// one lane per particle that walks its list with one warp or less to a scheduler. Here a stage
// boundary is one grid barrier, a particle's state and list stay on chip, and a team of LANES
// lanes evaluates its pairs, each lane its share. The sums stay in list order: the pair terms go
// through shared memory as the two factors of each accumulator's fused multiply-add, and one lane
// per accumulator runs it over them. The arithmetic and its order are those of the per-phase
// kernels (pbf_step.cuh, pbf_nbr.cuh): the same bits.
//
// Barrier: a counter that every block adds one to; thread 0 of a block waits until the count
// reaches the stage's target. A wait gives up after a bounded number of reads, sets
// PBF_ERRBIT_TIMEOUT and returns (the launch is cooperative, so every block is resident and a
// wait ends). No block passes a barrier that another one has not reached, so a launch that gives up
// leaves its memory in bounds, but the counter and the cell counts stay as they are: a launch that
// finds the bit set returns before its first write. The last block to leave sets the counter back
// to zero.
#include <cstdint>

#include "pbf_device.cuh"
#include "pbf_nbr.cuh"
#include "pbf_small_form.h"
#include "pbf_step.cuh"

namespace pbf {
namespace {

constexpr uint32_t kScanTile = kSmallTile;             // cells; scan_tmp has an entry per tile
constexpr uint32_t kMaxSortedCell = 4096;              // larger cells keep the atomic order (as k_cellsort_big)
constexpr int kOwnEntries = 64;                        // list entries of a particle kept on chip
constexpr int kMaxSums = 5;                            // accumulators of one walk over a list
constexpr int kRounds = 4;                             // pairs a lane evaluates between two exchanges
constexpr uint32_t kDirectTiles = 16;                  // tiles up to which a block sums the counts before its own
constexpr unsigned kMaxPolls = 1u << 22;             // reads of the barrier's counter (Buffers::wait_reads 0)

struct SmallStep {
  const float4 *pos_a, *vel_a;
  const uint32_t* id_a;
  float4 *pos_b, *vel_b, *disp, *xs0, *xs1, *pred;
  uint32_t* id_b;
  float *rho, *rho_iter0;
  uint32_t *count, *start, *tile, *xkey, *idkey;
  uint4* hdr;
  uint32_t* words;
  const SceneDesc* scenes;
  unsigned *err, *bar;
  unsigned polls;
  uint32_t m;
  int n, iters;
  float dt, inv_dt, one;
};

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, unsigned polls, unsigned* err) {
  __shared__ bool passed;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    unsigned seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
    } while (seen < target && --polls > 0);
    passed = seen >= target;
    if (!passed) atomicOr(err, PBF_ERRBIT_TIMEOUT);
  }
  __syncthreads();
  return passed;
}

// The same between the blocks of a cluster, in hardware. There every block keeps x* and the
// displacements of the whole scene in its shared memory: a particle's team stores what it computes
// into all blocks, and the neighbours' values are local loads.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// dst: an address of this block's shared memory; v goes to it in blocks u, u + LANES, ... of the
// cluster.
template <int LANES>
__device__ __forceinline__ void put_all(const void* dst, const float4& v, int u, unsigned blocks) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  for (unsigned r = u; r < blocks; r += LANES) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
  }
}

// Exclusive scan over the block's threads; *total is the sum.
template <int T>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* total) {
  constexpr int kWarps = T / 32;
  __shared__ uint32_t sums[kWarps];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= static_cast<unsigned>(o)) x += y;
  }
  __syncthreads();  // the sums of the call before are read
  if (lane == 31) sums[warp] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < static_cast<int>(warp)) before += sums[w];
    all += sums[w];
  }
  *total = all;
  return before + x - v;
}

// One lane per particle: calls f(load(j)) for every neighbour of a list in order, 8 gathers ahead
// of the arithmetic. quad(g): the 16 bytes of entries 8 g to 8 g + 7.
template <typename T, typename Q, typename L, typename F>
__device__ __forceinline__ void lane_walk(const uint4& h, Q&& quad, L&& load, F&& f) {
  const int total = nbr_total(h);
  T t[8];
  for (int g = 0; 8 * g < total; ++g) {
    const uint4 q = quad(g);
    const uint32_t e[8] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16,
                           q.z & 0xffffu, q.z >> 16, q.w & 0xffffu, q.w >> 16};
    if (8 * g + 8 <= total) {
#pragma unroll
      for (int u = 0; u < 8; ++u) t[u] = load(nbr_decode(h, e[u]));
#pragma unroll
      for (int u = 0; u < 8; ++u) f(t[u]);
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (8 * g + u < total) t[u] = load(nbr_decode(h, e[u]));
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (8 * g + u < total) f(t[u]);
    }
  }
}

// A team's walk over its particle's list. load(e) fetches what entry e needs, terms(x, o) gives
// the factors o[a].x, o[a].y of accumulator a's fused multiply-add; lane a % LANES of the team
// adds them in list order into acc[a / LANES]. buf: the team's shared memory. total: the list's
// length, most: the longest of the warp. All lanes of the warp call it.
template <int LANES, int NSUM, typename T, typename L, typename F>
__device__ __forceinline__ void team_sums(float (&acc)[(NSUM + LANES - 1) / LANES], float2* buf, int total, int most,
                                          L&& load, F&& terms) {
  constexpr int CH = LANES * kRounds, ROW = CH + 1, MINE = (NSUM + LANES - 1) / LANES;
  const int u = static_cast<int>(lane_id()) & (LANES - 1);
  T t[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (r * LANES + u < total) t[r] = load(r * LANES + u);
  for (int c = 0; c < most; c += CH) {
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int e = r * LANES + u;
      if (c + e < total) {
        float2 o[NSUM];
        terms(t[r], o);
#pragma unroll
        for (int a = 0; a < NSUM; ++a) buf[a * ROW + e] = o[a];
      }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int e = c + CH + r * LANES + u;
      if (e < total) t[r] = load(e);
    }
    const int m = min(CH, total - c);
#pragma unroll
    for (int q = 0; q < MINE; ++q) {
      const int a = q * LANES + u;
      if (a < NSUM) {
        const float2* row = buf + a * ROW;
        for (int k = 0; k < m; k += 8) {
          float2 w[8];
#pragma unroll
          for (int z = 0; z < 8; ++z) w[z] = row[min(k + z, CH - 1)];
#pragma unroll
          for (int z = 0; z < 8; ++z)
            if (k + z < m) acc[q] = __fmaf_rn(w[z].x, w[z].y, acc[q]);
        }
      }
    }
    __syncwarp();
  }
}

// Accumulator a of the team, in all its lanes.
template <int LANES, int M>
__device__ __forceinline__ float team_get(const float (&acc)[M], int a) {
  return __shfl_sync(0xffffffffu, acc[a / LANES], a & (LANES - 1), LANES);
}

template <int T, int LANES, bool CLUSTER>
constexpr size_t small_smem() {
  if (LANES == 1) return sizeof(NbrWarp) * (T / 32);  // the lists take the tables' place
  const size_t lists = sizeof(uint16_t) * kOwnEntries * (T / LANES);
  const size_t bufs = sizeof(float2) * kMaxSums * (LANES * kRounds + 1) * (T / LANES);
  const size_t tables = sizeof(NbrWarp) * (T / LANES / 32);
  const size_t copies = CLUSTER ? 3 * sizeof(float4) * kClusterBlocks * (T / LANES) : 0;
  return copies + lists + (bufs > tables ? bufs : tables);
}

// T threads a block. The first T / LANES of them also take one particle each in the stages before
// the iterations: prediction, sort, neighbour build.
// CLUSTER: the grid is one thread block cluster and the barrier the cluster's own.
template <int T, int LANES, bool N4, bool CLUSTER>
__global__ void __launch_bounds__(T, 512 / T) k_step_small(const __grid_constant__ SmallStep A,
                                                            const __grid_constant__ DevParams P) {
  constexpr int kScanItems = static_cast<int>(kScanTile) / T;
  constexpr int PB = T / LANES;  // particles of a block
  extern __shared__ uint4 smem[];
  constexpr int kCopy = CLUSTER ? static_cast<int>(kClusterBlocks) * PB : 0;  // particles of a cluster
  float4* copies = reinterpret_cast<float4*>(smem);
  uint16_t* lists = reinterpret_cast<uint16_t*>(copies + 3 * kCopy);
  char* work = reinterpret_cast<char*>(lists + (LANES == 1 ? 0 : kOwnEntries * PB));
  const unsigned full = 0xffffffffu;
  const unsigned G = gridDim.x;
  const int tid = static_cast<int>(threadIdx.x);
  const int n = A.n;
  unsigned target = 0;
#define PBF_GRID_BARRIER()                                       \
  if constexpr (CLUSTER)                                         \
    cluster_barrier();                                           \
  else if (!grid_barrier(A.bar, target += G, A.polls, A.err))             \
    return

  // prediction (particles.cpp:175-183, 87-132) and cell counts
  const int i = static_cast<int>(blockIdx.x) * PB + tid;
  const bool front = tid < PB;  // whole warps
  const bool live = front && i < n;
  float4 x4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float3 d = make_float3(0.f, 0.f, 0.f), xp = d;
  uint32_t key = 0xffffffffu, id = 0u, rank = 0u;
  if (live) {
    x4 = A.pos_a[i];
    id = A.id_a[i];
  }
  // a step before gave up: its barrier and counts are unusable (read beside the particles)
  if constexpr (!CLUSTER) {
    if (__syncthreads_or(static_cast<int>(__ldcg(A.err) & PBF_ERRBIT_TIMEOUT))) return;
  }
  if (live) {
    const SceneDesc& sc = A.scenes[scene_of_slot(x4)];
    const float3 x = f3(x4);
    collide<false, false>(x, d, predict_delta(A.vel_a[i], P, A.dt), true, sc, P);
    xp = displaced(x, d);
    key = cell_key(cell_of(xp, sc, P.inv_cell), sc);
  }
  if (front) rank = count_rank(key, live, A.count);  // the counts are zero between steps
  PBF_GRID_BARRIER();

  // Exclusive scan of the counts, tile by tile. With few tiles a block sums the counts of all
  // tiles before its own itself; with more the tiles' sums are exchanged, one barrier later.
  const uint32_t tiles = (A.m + kScanTile - 1) / kScanTile;
  const bool direct = tiles <= kDirectTiles && tiles <= G;
  for (uint32_t t = blockIdx.x; t < tiles; t += G) {
    const uint32_t base = t * kScanTile + tid * kScanItems;
    uint32_t v[kScanItems], s = 0, total, before = 0;
    if (direct) {
      const uint4* c4 = reinterpret_cast<const uint4*>(A.count);
      for (uint32_t c = tid; c < t * (kScanTile / 4); c += T) {
        const uint4 q = c4[c];
        before += q.x + q.y + q.z + q.w;
      }
      block_scan<T>(before, &before);
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = base + k < A.m ? A.count[base + k] : 0u;
      s += v[k];
    }
    uint32_t off = before + block_scan<T>(s, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < A.m) A.start[base + k] = off;
      off += v[k];
    }
    if (tid == 0) {
      A.tile[t] = total;
      if (t == tiles - 1 && direct) A.start[A.m] = before + total;
    }
  }
  PBF_GRID_BARRIER();
  for (uint32_t c = blockIdx.x * T + tid; c < A.m; c += G * T) A.count[c] = 0u;  // for the next step
  if (!direct) {
    for (uint32_t t = blockIdx.x; t < tiles; t += G) {
      uint32_t s = 0, before;
      for (uint32_t u = tid; u < t; u += T) s += A.tile[u];
      block_scan<T>(s, &before);
      const uint32_t base = t * kScanTile + tid * kScanItems;
      if (before) {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
          if (base + k < A.m) A.start[base + k] += before;
      }
      if (t == tiles - 1 && tid == 0) A.start[A.m] = before + A.tile[t];
    }
    PBF_GRID_BARRIER();
  }

  // cell order: by x of x*, then original index (as k_cellrank and k_cellsort_big); the slot's
  // state goes there at once
  uint32_t cb = 0, ce = 0;
  const uint32_t xkey = order_bits(xp.x);
  if (live) {
    cb = A.start[key];
    ce = A.start[key + 1];
    A.xkey[cb + rank] = xkey;
    A.idkey[cb + rank] = id;
  }
  PBF_GRID_BARRIER();
  if (live) {
    uint32_t r = rank;
    if (ce - cb <= kMaxSortedCell) {
      const uint64_t mine = (static_cast<uint64_t>(xkey) << 32) | id;
      r = 0;
#pragma unroll 4
      for (uint32_t u = cb; u < ce; ++u)
        r += ((static_cast<uint64_t>(A.xkey[u]) << 32) | A.idkey[u]) < mine ? 1u : 0u;
    }
    const uint32_t s = cb + r;
    A.pos_b[s] = x4;
    A.id_b[s] = id;
    A.disp[s] = make_float4(d.x, d.y, d.z, 0.f);
    const float4 xs = make_float4(xp.x, xp.y, xp.z, 0.f);
    A.xs0[s] = xs;
    if (A.pred) A.pred[s] = xs;
  }
  PBF_GRID_BARRIER();

  // neighbour lists of the block's slots
  float4 *cur = A.xs0, *nxt = A.xs1, *disp = A.disp;
  if constexpr (CLUSTER) {
    cur = copies;
    nxt = copies + kCopy;
    disp = copies + 2 * kCopy;
    for (int j = tid; j < n; j += T) {
      cur[j] = A.xs0[j];
      disp[j] = A.disp[j];
    }
  }
  if (front)
    nbr_build_warp<false, false>(reinterpret_cast<NbrWarp*>(work)[tid >> 5], i, A.xs0, A.pos_b, A.start, A.scenes, A.hdr,
                          A.words, A.err, P, A.one, n);
  if constexpr (CLUSTER)
    cluster_barrier();  // every block has its copies before another one stores into them
  else
    __syncthreads();

  // from here on a team of LANES lanes holds slot p
  const int team = tid / LANES, u = tid & (LANES - 1);
  const int p = static_cast<int>(blockIdx.x) * PB + team;
  const bool act = p < n, lead = act && u == 0;
  constexpr int kOwnQuads = static_cast<int>(sizeof(NbrWarp) / (32 * sizeof(uint4)));
  uint16_t* own = lists + kOwnEntries * team;
  const uint16_t* entries = reinterpret_cast<const uint16_t*>(A.words);
  uint4* own4 = reinterpret_cast<uint4*>(reinterpret_cast<NbrWarp*>(work) + (tid >> 5)) + lane_id();  // LANES 1
  const uint4* far4 = reinterpret_cast<const uint4*>(A.words) + p;
  uint4 h = make_uint4(0u, 0u, 0u, 0u);
  float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
  x4 = xi;
  d = make_float3(0.f, 0.f, 0.f);
  if (act) {
    h = A.hdr[p];
    x4 = A.pos_b[p];
    xi = cur[p];
    d = f3(disp[p]);
  }
  const int total = nbr_total(h);
  const int most = __reduce_max_sync(full, total);
  auto far = [&](int e) -> uint16_t { return entries[8 * (static_cast<size_t>(e >> 3) * n + p) + (e & 7)]; };
  if constexpr (LANES == 1) {
    for (int g = 0; g < kOwnQuads && 8 * g < total; ++g) own4[32 * g] = far4[static_cast<size_t>(g) * n];
  } else {
    for (int e = u; e < min(total, kOwnEntries); e += LANES) own[e] = far(e);
  }
  __syncwarp();
  auto quad = [&](int g) -> uint4 { return g < kOwnQuads ? own4[32 * g] : far4[static_cast<size_t>(g) * n]; };
  auto slot = [&](int e) -> uint32_t { return nbr_decode(h, e < kOwnEntries ? own[e] : far(e)); };
  float2* buf = reinterpret_cast<float2*>(work) + kMaxSums * (LANES * kRounds + 1) * team;
  const SceneDesc& sc = A.scenes[act ? scene_of_slot(x4) : 0];
  const float wt = P.poly6_c * P.tis;

  // Jacobi iterations (particles.cpp:185-213). The first lambda pass needs no barrier: it reads
  // what the build read, and writes only its own x*.w.
  auto load_x = [&](int e) -> float4 { return cur[slot(e)]; };
  for (int it = 0; it < A.iters; ++it) {
    {
      LambdaSum sum;
      if constexpr (LANES == 1) {
        lane_walk<float4>(h, quad, [&](uint32_t j) { return cur[j]; },
                          [&](const float4& xj) { sum.add(xi, xj, P); });
      } else {
        float acc[(5 + LANES - 1) / LANES] = {};
        team_sums<LANES, 5, float4>(acc, buf, total, most, load_x, [&](const float4& xj, float2* o) {
          const Pair q = pair_of(xi, xj, P.h, P.h2);
          o[0] = make_float2(__fmul_rn(q.q, q.q), q.q);
          o[1] = make_float2(__fmul_rn(q.s, q.s), q.r2);
          o[2] = make_float2(q.r.x, q.s);
          o[3] = make_float2(q.r.y, q.s);
          o[4] = make_float2(q.r.z, q.s);
        });
        sum.qsum = team_get<LANES>(acc, 0);
        sum.g2 = team_get<LANES>(acc, 1);
        sum.gs = make_float3(team_get<LANES>(acc, 2), team_get<LANES>(acc, 3), team_get<LANES>(acc, 4));
      }
      float rho;
      xi.w = sum.lambda(P, &rho);
      if (CLUSTER && act) put_all<LANES>(&cur[p], xi, u, G);
      if (lead) {
        if (!CLUSTER) cur[p].w = xi.w;
        if (it == 0 && A.rho_iter0) A.rho_iter0[p] = rho;
      }
    }
    PBF_GRID_BARRIER();
    {
      DeltaSum<N4> sum;
      if constexpr (LANES == 1) {
        lane_walk<float4>(h, quad, [&](uint32_t j) { return cur[j]; },
                          [&](const float4& xj) { sum.add(xi, xj, wt, P); });
      } else {
        float acc[(3 + LANES - 1) / LANES] = {};
        team_sums<LANES, 3, float4>(acc, buf, total, most, load_x, [&](const float4& xj, float2* o) {
          float c;
          const float3 r = delta_term<N4>(xi, xj, wt, P, &c);
          o[0] = make_float2(r.x, c);
          o[1] = make_float2(r.y, c);
          o[2] = make_float2(r.z, c);
        });
        sum.dp = make_float3(team_get<LANES>(acc, 0), team_get<LANES>(acc, 1), team_get<LANES>(acc, 2));
      }
      if (act) {
        const float3 x = f3(x4);
        collide<false, false>(x, d, sum.delta(P), false, sc, P);
        const float3 xn = displaced(x, d);
        xi = make_float4(xn.x, xn.y, xn.z, 0.f);
        const float4 d_out = make_float4(d.x, d.y, d.z, 0.f);
        if (CLUSTER) {
          put_all<LANES>(&nxt[p], xi, u, G);
          if (it == A.iters - 1) put_all<LANES>(&disp[p], d_out, u, G);
        } else if (lead) {
          nxt[p] = xi;
          if (it == A.iters - 1) disp[p] = d_out;
        }
      }
    }
    PBF_GRID_BARRIER();
    float4* t = cur;
    cur = nxt;
    nxt = t;
  }

  // velocity, vorticity, XSPH, density; then vorticity confinement, x <- x* (particles.cpp:215-248)
  const float3 vi = d * A.inv_dt;
  auto load_xd = [&](int e) {
    const uint32_t j = slot(e);
    return XD{cur[j], disp[j]};
  };
  XsphSum xs;
  if constexpr (LANES == 1) {
    lane_walk<XD>(h, quad, [&](uint32_t j) { return XD{cur[j], disp[j]}; },
                  [&](const XD& q) { xs.add(xi, vi, q, A.inv_dt, P); });
  } else {
    float acc[(4 + LANES - 1) / LANES] = {};
    team_sums<LANES, 4, XD>(acc, buf, total, most, load_xd, [&](const XD& a, float2* o) {
      const XsphTerm q = xsph_term(xi, vi, a, A.inv_dt, P);
      o[0] = make_float2(q.vij.x, q.q3);
      o[1] = make_float2(q.vij.y, q.q3);
      o[2] = make_float2(q.vij.z, q.q3);
      o[3] = make_float2(q.q3, 1.0f);
    });
    xs.visc = make_float3(team_get<LANES>(acc, 0), team_get<LANES>(acc, 1), team_get<LANES>(acc, 2));
    xs.qsum = team_get<LANES>(acc, 3);
  }
  if constexpr (LANES > 1) {
    float acc[(3 + LANES - 1) / LANES] = {};
    team_sums<LANES, 3, XD>(acc, buf, total, most, load_xd, [&](const XD& a, float2* o) {
      const XsphTerm q = xsph_term(xi, vi, a, A.inv_dt, P);
      o[0] = make_float2(q.w.x, 1.0f);
      o[1] = make_float2(q.w.y, 1.0f);
      o[2] = make_float2(q.w.z, 1.0f);
    });
    xs.w = make_float3(team_get<LANES>(acc, 0), team_get<LANES>(acc, 1), team_get<LANES>(acc, 2));
  }
  const float4 w = xs.omega(P);
  if (CLUSTER && act) put_all<LANES>(&cur[p], make_float4(xi.x, xi.y, xi.z, w.w), u, G);
  if (lead) {
    if (!CLUSTER) cur[p].w = w.w;
    A.rho[p] = xs.rho(P);
  }
  PBF_GRID_BARRIER();
  {
    VortSum sum;
    if constexpr (LANES == 1) {
      lane_walk<float4>(h, quad, [&](uint32_t j) { return cur[j]; },
                        [&](const float4& xj) { sum.add(xi, xj, P); });
    } else {
      float acc[(3 + LANES - 1) / LANES] = {};
      team_sums<LANES, 3, float4>(acc, buf, total, most, load_x, [&](const float4& xj, float2* o) {
        float c;
        const float3 r = vort_term(xi, xj, P, &c);
        o[0] = make_float2(r.x, c);
        o[1] = make_float2(r.y, c);
        o[2] = make_float2(r.z, c);
      });
      sum.eta = make_float3(team_get<LANES>(acc, 0), team_get<LANES>(acc, 1), team_get<LANES>(acc, 2));
    }
    if (lead) {
      const float3 v = confined(xs.velocity(vi, P), sum.location(P), w, A.dt, P);
      A.vel_b[p] = make_float4(v.x, v.y, v.z, 0.f);
      A.pos_b[p] = make_float4(xi.x, xi.y, xi.z, x4.w);
      if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z)))
        atomicOr(A.err, PBF_ERRBIT_NONFINITE);
    }
  }
#undef PBF_GRID_BARRIER
  // every block is past the last barrier when it counts itself out; the last one clears the count
  if (!CLUSTER && tid == 0 && atomicInc(A.bar + 1, G - 1) == G - 1) *A.bar = 0u;
}

using Kernel = void (*)(SmallStep, DevParams);
template <int T, int LANES, bool CLUSTER>
Kernel pick_kernel(bool n4) {
  return n4 ? k_step_small<T, LANES, true, CLUSTER> : k_step_small<T, LANES, false, CLUSTER>;
}
struct Form {
  Kernel kernel;
  SmallFormSize size;
  size_t smem;
};
Form pick(int form, bool n4) {
  const SmallFormSize& z = kSmallForm[form];
  switch (form) {
    case 1: return Form{pick_kernel<512, 8, true>(n4), z, small_smem<512, 8, true>()};
    case 2: return Form{pick_kernel<256, 8, false>(n4), z, small_smem<256, 8, false>()};
    case 3: return Form{pick_kernel<128, 1, false>(n4), z, small_smem<128, 1, false>()};
    default: return Form{pick_kernel<256, 1, false>(n4), z, small_smem<256, 1, false>()};
  }
}

void set_config(const Form& f, uint32_t blocks, cudaStream_t s, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(blocks);
  cfg->blockDim = dim3(f.size.threads);
  cfg->dynamicSmemBytes = f.smem;
  cfg->stream = s;
  *at = cudaLaunchAttribute{};
  if (f.size.cluster) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = blocks;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
  } else {
    at->id = cudaLaunchAttributeCooperative;
    at->val.cooperative = 1;
  }
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// Whether the device takes the form: its launch can be resident. An error is an answer too (a device
// or a partition of one without clusters of 16 blocks, or with less shared memory): the next form.
bool takes(int form, bool n4) {
  const Form f = pick(form, n4);
  int fit = 0;
  cudaError_t e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(f.smem));
  if (e == cudaSuccess && f.size.cluster) {
    e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    set_config(f, kClusterBlocks, nullptr, &cfg, &at);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fit, f.kernel, &cfg);
  } else if (e == cudaSuccess) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, f.kernel, static_cast<int>(f.size.threads), f.smem);
    fit /= static_cast<int>(f.size.on_sm);
  }
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e == cudaSuccess && fit >= 1;
}

}  // namespace

// The kernels are looked at until one is taken, mostly the first: each look costs a handle's creation
// tens of microseconds, and the first one loads the kernel. Handles with collider triangles or spheres
// keep the per-phase kernels: whether a move meets a triangle's edge turns on the last bit, and the
// primitives' tests are not pinned to one rounding.
void small_step_setup(int device, const DevParams& P, Buffers* b) {
  int sms = 0, coop = 0;
  b->small_form = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    return;
  }
  b->small_form = small_form_for(b->n, b->n_cells, static_cast<size_t>(sms),
                                 [&](int form) { return takes(form, P.scorr_n == 4); });
}

int small_step_form(const Buffers& b, const DevParams& P) { return P.n_mesh > 0 || P.n_sph > 0 ? 0 : b.small_form; }

bool small_step_waits(int form) { return form != 0 && !kSmallForm[form].cluster; }

cudaError_t launch_step_small(const Buffers& b, const DevParams& P, int form, int cur, float dt, int iters,
                              bool keep_pred, cudaStream_t s) {
  const int A = cur, B = 1 - cur;
  SmallStep a{};
  a.pos_a = b.pos[A];
  a.vel_a = b.vel[A];
  a.id_a = b.id[A];
  a.pos_b = b.pos[B];
  a.vel_b = b.vel[B];
  a.id_b = b.id[B];
  a.disp = b.disp[1];
  a.xs0 = b.xs[0];
  a.xs1 = b.xs[1];
  a.pred = keep_pred ? b.pred : nullptr;
  a.rho = b.rho;
  a.rho_iter0 = P.stats ? b.rho_iter0 : nullptr;
  a.count = b.cell_count;
  a.start = b.cell_start;
  a.tile = b.scan_tmp;
  a.xkey = b.perm_atomic;
  a.idkey = b.perm;
  a.hdr = b.nbr_hdr;
  a.words = b.nbr_w;
  a.scenes = b.scenes;
  a.err = b.err;
  a.bar = b.grid_bar;
  a.polls = b.wait_reads ? b.wait_reads : kMaxPolls;
  a.m = b.n_cells;
  a.n = static_cast<int>(b.n);
  a.iters = iters;
  a.dt = dt;
  a.inv_dt = 1.0f / dt;
  a.one = 1.0f;
  const uint32_t tiles = (a.m + kScanTile - 1) / kScanTile;
  const Form f = pick(form, P.scorr_n == 4);
  const uint32_t need = (static_cast<uint32_t>(b.n) + f.size.per_block - 1) / f.size.per_block;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  set_config(f, need > tiles ? need : tiles, s, &cfg, &at);
  return cudaLaunchKernelEx(&cfg, f.kernel, a, P);
}

}  // namespace pbf
