// The neighbour build (particles.cpp:258-265): the warp scan and the thread scan, shared by the
// per-phase kernel (pbf_kernels.cu) and the whole-step kernel of small scenes (pbf_small.cu).
#pragma once

#include <cmath>
#include <cstdint>

#include "pbf_device.cuh"

namespace pbf {

__device__ __forceinline__ int scene_of_slot(const float4& p) { return __float_as_int(p.w); }

// NC: through the read-only path, for data that no thread writes during the kernel.
template <bool NC, typename T>
__device__ __forceinline__ T ld(const T* p) {
  return NC ? __ldg(p) : *p;
}

// One thread scans one particle's candidates: for the warps whose slots lie far apart (in many rows,
// or along them), that are next to a cell too large to be sorted, or whose list offsets pass their 14
// bits; in the whole-step kernel also where windows exceed the shared tables. Each of the
// 9 candidate rows (3 z-slabs x 3 y-rows) is skipped when its cells lie beyond h in y/z, and
// otherwise trimmed in x to the cells that reach [x - w, x + w], w = sqrt(h^2 - d_yz^2): about
// 20 of the 27 cells on average. Within the trimmed row (sorted by x, see k_cellrank) only
// candidates with |dx| <= w are tested. All tests keep a margin of 1e-3 cell, far above the
// FP32 rounding of the cell binning and of the predicate, so no pair within h is dropped.
template <bool NC>
__device__ __noinline__ void nbr_scan_thread(int i, const float4* xs, const float4* pos, const uint32_t* cell_start,
                                             const SceneDesc* __restrict__ scenes, uint4* hdr, uint32_t* words,
                                             unsigned* err, const DevParams& P, int n) {
  const float4 xi = xs[i];
  const SceneDesc& sc = scenes[scene_of_slot(pos[i])];
  const CellCoord cc = cell_of(f3(xi), sc, P.inv_cell);
  const int cap = P.max_words * 2;
  uint32_t gbase[3] = {0u, 0u, 0u};
  int total = 0;
  // List entries are stored one 16-bit half-word at a time: entry k of the slot is
  // half-word k % 8 of its group k / 8 (list_word's word k / 2, low half first), so an
  // append is one straight path with no word to assemble. (Pairing entries into words before
  // storing: 0.232 against 0.210 ms; collecting a group in registers or in shared memory and
  // storing it as one 16-byte write measured slower still: the appends run divergently, and
  // extra instructions and a smaller L1 cost more than coalesced stores save.)
  uint16_t* eptr = reinterpret_cast<uint16_t*>(words) + 8 * static_cast<size_t>(i);
  const size_t estep = 8 * static_cast<size_t>(n) - 7;
  unsigned flags = 0;
  // position inside the own cell, in cells, and the reach in cells with its margin
  const float fy = (xi.y - sc.origin[1]) * P.inv_cell - static_cast<float>(cc.y);
  const float fz = (xi.z - sc.origin[2]) * P.inv_cell - static_cast<float>(cc.z);
  const float m = 1e-3f;
  const float reach = sqrtf(P.h2) * P.inv_cell + m;
  const float reach2 = reach * reach;
  const float ux = (xi.x - sc.origin[0]) * P.inv_cell;
  const float cell_w = 1.0f / P.inv_cell;
  const int y0 = cc.y > 0 ? cc.y - 1 : 0;
  const float2 nxy = make_float2(-xi.x, -xi.y);
  const float nz = -xi.z;
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const int z = cc.z + g - 1;
    if (z < 0 || z >= sc.dim[2]) continue;
    const uint32_t slab = sc.cell_off + static_cast<uint32_t>(z * sc.dim[1] * sc.dim[0]);
    const int x0 = cc.x > 0 ? cc.x - 1 : 0;
    gbase[g] = ld<NC>(&cell_start[slab + static_cast<uint32_t>(y0 * sc.dim[0] + x0)]);
    const float dz = g == 0 ? fmaxf(fz - m, 0.f) : (g == 2 ? fmaxf(1.f - fz - m, 0.f) : 0.f);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int y = cc.y + r - 1;
      if (y < 0 || y >= sc.dim[1]) continue;
      const float dy = r == 0 ? fmaxf(fy - m, 0.f) : (r == 2 ? fmaxf(1.f - fy - m, 0.f) : 0.f);
      const float w2 = reach2 - (dy * dy + dz * dz);
      if (w2 < 0.f) continue;
      const float w = sqrtf(w2);
      const int xa = max(max(static_cast<int>(floorf(ux - w)), cc.x - 1), 0);
      const int xb = min(min(static_cast<int>(floorf(ux + w)), cc.x + 1), sc.dim[0] - 1);
      if (xa > xb) continue;
      const uint32_t row = slab + static_cast<uint32_t>(y * sc.dim[0]);
      const uint32_t start = ld<NC>(&cell_start[row + xa]);
      uint32_t end = ld<NC>(&cell_start[row + xb + 1]);
      if (end - start > static_cast<uint32_t>(kMaxRowCandidates)) {
        flags |= PBF_ERRBIT_ROW_CAPACITY;
        end = start + kMaxRowCandidates;
      }
      const uint32_t gb = gbase[g];
      const uint32_t gbits = static_cast<uint32_t>(g) << kOffsetBits;
      // the row is sorted by x: a binary search over the window's first cell (the only
      // one reaching below x - W) finds the first candidate at or above x - W, and the
      // first one above x + W ends the row (W = w cells, margin included; with NaN
      // coordinates in the cell the search may start early, never late). The predicate
      // reuses the x difference. Every difference and square is rounded, |x*_i - x*_j|^2 <= H2
      // of particles.cpp:260 as a host check repeats it. The own slot is a hit at
      // distance 0 and is dropped there, which keeps one loop per row (two half-row loops
      // around it: 0.209 against 0.206 ms; one loop over a slab's three rows, lanes moving
      // on to the next row when theirs ends: 0.243 against 0.234 ms, 48 registers).
      const uint32_t ui = static_cast<uint32_t>(i);
      const float W = w * cell_w;
      const uint32_t first_end = ld<NC>(&cell_start[row + xa + 1]);
      uint32_t a = start, hi = min(end, first_end);
      while (a < hi) {
        const uint32_t md = (a + hi) >> 1;
        if (ld<NC>(&xs[md].x) - xi.x < -W) a = md + 1; else hi = md;
      }
      for (uint32_t j = a; j < end; ++j) {
        const float4 xj = ld<NC>(&xs[j]);
        // x and y of x*_j - x*_i as one packed FP32x2 add against -x*_i (negation is
        // exact: the same roundings as x*_i - x*_j up to sign) and one packed square
        const float2 dxy = __fadd2_rn(make_float2(xj.x, xj.y), nxy);
        if (dxy.x > W) break;
        const float2 sq = __fmul2_rn(dxy, dxy);
        const float dz = __fadd_rn(xj.z, nz);
        if (__fadd_rn(__fadd_rn(sq.x, sq.y), __fmul_rn(dz, dz)) <= P.h2 && j != ui) {
          const uint32_t off = j - gb;
          if (off <= kOffsetMask && total < cap) {
            *eptr = static_cast<uint16_t>(gbits | off);
            eptr += ((total & 7) == 7) ? estep : 1;
            ++total;
          } else {
            flags |= off > kOffsetMask ? PBF_ERRBIT_ROW_CAPACITY : PBF_ERRBIT_NEIGHBOR_CAPACITY;
          }
        }
      }
    }
  }
  // the slab bases relative to slab 0's, less the tag bits (nbr_decode)
  hdr[i] = make_uint4(gbase[0], gbase[1] - gbase[0] - (1u << kOffsetBits),
                      gbase[2] - gbase[0] - (2u << kOffsetBits), static_cast<uint32_t>(total));
  if (flags) atomicOr(err, flags);
}

// A warp scans the candidates of its 32 consecutive slots together. The slots are split into
// groups: the slots of one grid row within 8 aligned ones. A group's slots ascend in x, so
// the candidates of all of them are, in each of the 9 rows around theirs, one slot range (cells
// one before the first to one after the last, trimmed by binary search to the x reach). The
// ranges are read as one flat list, 32 candidates a turn, one per lane; a turn tests its 32
// candidates against the group's slots, two slots at a time in packed FP32x2 (the thread
// scan's roundings), and each slot's 32 results are one ballot word in shared memory. Then each lane
// turns the words of its own slot into list entries, in ascending slot order as the thread scan
// appends them, all lanes at the same entry index: 8 entries make one 16-byte store, and a warp's
// stores are contiguous. The lists (neighbours and their order) are the thread scan's.
//
// Why: with one particle per lane the scan is a serial chain of dependent loads whose windows
// differ from lane to lane (53% of lanes active, 193 warp instructions a particle). Here every
// lane has a candidate in every turn and a candidate is loaded once for 8 particles; the window
// of 8 slots is wider than one particle's own (about 216 candidates against 91 at rest spacing),
// which the packed tests more than pay for. 1M colliding blocks: 234 -> 175 us a build, 150M
// warp instructions instead of 202M; 33k particles at 46 neighbours 62 -> 31 us; 720 particles
// 27 -> 18 us. Of the 175 us about 25 are the list entries, 40 the tests, 26 the candidate loads,
// 22 the binary searches, the rest the turns' and the groups' bookkeeping. Measured and rejected:
// the slots held in registers (64 a thread, 5 us more), candidates loaded a turn ahead and middle
// rows left untrimmed (193 us).
constexpr int kNbrWords = 14;    // ballot words per slot: at most 448 candidates a group
constexpr int kNbrEntries = 1408;  // candidates of the groups of a round, each group's rounded up to 32
// The thread scan takes the warps of more groups than the tables hold (slots scattered over rows),
// and those whose groups' windows are so many cells long in all that a lane has few candidates of
// its own in them: 0.13 particles a cell 33.8 us with the group scan, 30.0 with the thread scan; 0.5
// a cell (80 to 100 cells) 96 and 110; rest spacing has about 18 cells, 1 particle a cell 55.
constexpr int kNbrGroups = 6;
constexpr int kNbrSpan = 160;
struct NbrWarp {
  uint32_t mask[kNbrWords][32];   // [turn][slot]: the turn's 32 candidates within h of the slot
  float4 txy[16];                 // slots 2p and 2p + 1: -x, -x, -y, -y
  float2 tz[16];                  // -z, -z
  int2 de[9];                     // the current group's non-empty rows: candidate slot less flat index; entry less slot
  uint4 row[9 * kNbrGroups];      // per (group, row): first candidate slot, count, entry less slot
  uint32_t gb[3 * kNbrGroups];    // the slabs' first slots
  int first[kNbrGroups + 1];      // first lane per group; after the last, the live lanes
  int cand[kNbrGroups];           // candidates per group
  int eoff[kNbrGroups];           // their first entry in ent
  uint16_t ent[kNbrEntries + 32];  // list entry of every candidate; the last 32 are read, not used,
                                   // by lanes past their hits
};

enum NbrResult { kNbrDone, kNbrParts, kNbrThread };  // a warp's lists: made; left to PARTS; to the thread scan

// PARTS: a group with more candidates than the words hold is read in pieces, each appending to the
// lists of the pieces before (16-bit stores; clumps of 2.6 times the rest spacing's density and more:
// 262k particles at 93 neighbours 199 -> 154 us, at 114 neighbours 405 -> 254, by the thread scan
// before). A code of its own, behind the first try, because its registers cost the common case 0.5%.
template <bool NC, bool PARTS>
__device__ __forceinline__ NbrResult nbr_build_lists(NbrWarp& S, int i, const float4* xs, const float4* pos,
                                                     const uint32_t* cell_start, const SceneDesc* __restrict__ scenes,
                                                     uint4* hdr, uint32_t* words, unsigned* err, const DevParams& P,
                                                     float one, int n) {
  const unsigned full = 0xffffffffu;
  const int lane = static_cast<int>(lane_id());
  const bool live = i < n;
  const unsigned alive = __ballot_sync(full, live);  // a prefix of the lanes
  if (!alive) return kNbrDone;
  const unsigned upto = lane == 31 ? full : ((2u << lane) - 1u);
  const float2 ones = make_float2(one, one);  // 1, unknown to the compiler
  const float4 xi = live ? xs[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int scn = live ? scene_of_slot(pos[i]) : 0;
  uint32_t row0 = 0xffffffffu;
  CellCoord cc{0, 0, 0};
  if (live) {
    const SceneDesc& sc = scenes[scn];
    cc = cell_of(f3(xi), sc, P.inv_cell);
    row0 = sc.cell_off + static_cast<uint32_t>((cc.z * sc.dim[1] + cc.y) * sc.dim[0]);
  }
  const uint32_t prev = __shfl_up_sync(full, row0, 1);
  const bool head = live && ((lane & 7) == 0 || prev != row0);
  const unsigned heads = __ballot_sync(full, head);
  const int ng = __popc(heads), group = __popc(heads & upto) - 1;  // groups; the lane's
  if (!PARTS) {
    // cells along x of the groups' windows
    const unsigned above = heads & ~upto;
    const int last = (above ? __ffs(above) - 1 : __popc(alive)) - 1;
    const int span = __shfl_sync(full, cc.x, last) - cc.x + 3;
    if (ng > kNbrGroups || __reduce_add_sync(full, head ? span : 0) > kNbrSpan) return kNbrThread;
  }
  if (head) S.first[group] = lane;
  if (lane == 0) S.first[ng] = __popc(alive);
  const int p2 = lane >> 1, q2 = lane & 1;
  reinterpret_cast<float*>(&S.txy[p2])[q2] = -xi.x;
  reinterpret_cast<float*>(&S.txy[p2])[2 + q2] = -xi.y;
  reinterpret_cast<float*>(&S.tz[p2])[q2] = -xi.z;
  __syncwarp();
  // The candidate ranges, one (group, row) per lane and round: whole cells, trimmed in x to the
  // reach of the group's slots, h plus a margin of 1e-3 cell (NaN coordinates leave a range
  // untrimmed).
  bool ok = true, room = true;
  const float W = (sqrtf(P.h2) * P.inv_cell + 1e-3f) * (1.0f / P.inv_cell);
  for (int base = 0; base < 9 * ng; base += 32) {
    const int q = base + lane;
    const bool act = q < 9 * ng;
    const int s = act ? q / 9 : 0, r = act ? q - 9 * s : 0;
    const int f = S.first[s], l = S.first[s + 1] - 1;
    const int cy = __shfl_sync(full, cc.y, f), cz = __shfl_sync(full, cc.z, f);
    const int cxa = __shfl_sync(full, cc.x, f), cxb = __shfl_sync(full, cc.x, l);
    const float xa = __shfl_sync(full, xi.x, f), xb = __shfl_sync(full, xi.x, l);
    const int gs = __shfl_sync(full, scn, f);
    if (act) {
      const SceneDesc& sc = scenes[gs];
      const int d0 = sc.dim[0], d1 = sc.dim[1], d2 = sc.dim[2];
      const int g = r / 3, z = cz + g - 1, y = cy + (r - 3 * g) - 1;
      uint32_t lo = 0, lo2 = 0, gb = 0;
      if (z >= 0 && z < d2) {
        const uint32_t slab = sc.cell_off + static_cast<uint32_t>(z * d1 * d0);
        const int a = max(cxa - 1, 0), b = min(cxb + 1, d0 - 1);
        gb = ld<NC>(&cell_start[slab + static_cast<uint32_t>(max(cy - 1, 0) * d0 + a)]);
        if (y >= 0 && y < d1) {
          const uint32_t row = slab + static_cast<uint32_t>(y * d0);
          lo = ld<NC>(&cell_start[row + a]);
          lo2 = ld<NC>(&cell_start[row + b]);
          uint32_t hi = ld<NC>(&cell_start[row + a + 1]), hi2 = ld<NC>(&cell_start[row + b + 1]);
          if (hi2 - lo > static_cast<uint32_t>(kMaxRowCandidates)) ok = false;  // reported by the thread scan
          while (lo < hi || lo2 < hi2) {  // first x >= xa - W of the first cell; first x > xb + W of the last
            const uint32_t md = (lo + hi) >> 1, md2 = (lo2 + hi2) >> 1;
            if (lo < hi) {
              if (ld<NC>(&xs[md].x) - xa < -W) lo = md + 1; else hi = md;
            }
            if (lo2 < hi2) {
              if (ld<NC>(&xs[md2].x) - xb > W) hi2 = md2; else lo2 = md2 + 1;
            }
          }
        }
      }
      const uint32_t cnt = lo2 > lo ? lo2 - lo : 0u;
      if (cnt && lo2 - 1 - gb > kOffsetMask) ok = false;
      S.row[q] = make_uint4(lo, cnt, (static_cast<uint32_t>(g) << kOffsetBits) - gb, 0u);
      if (r == 3 * g + 1) S.gb[3 * s + g] = gb;
    }
  }
  __syncwarp();
  if (lane < ng) {  // lane s: group s
    uint32_t t = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) t += S.row[9 * lane + r].y;
    S.cand[lane] = static_cast<int>(t);
    if (!PARTS) room = t <= 32u * kNbrWords;
  }
  if (!__all_sync(full, ok)) return kNbrThread;
  if (!PARTS && !__all_sync(full, room)) return kNbrParts;
  __syncwarp();
  int s = 0, turn0 = 0;  // the next group and its first turn: a group beyond the words goes in pieces
  do {  // rounds of as many groups as the entries have room for (dense windows: fewer than all)
    const int s_begin = s, t_begin = turn0;
    int used = 0;
    for (; s < ng; ++s) {
      const int rest = S.cand[s] - 32 * turn0;
      const int T = min(rest, 32 * kNbrWords), eoff = used;
      if (used + T > kNbrEntries) break;
      const int f = S.first[s], l = S.first[s + 1] - 1;
      used += (T + 31) & ~31;
      if (lane == 0) S.eoff[s] = eoff;
      // lane r < 9: row r's range in the flat list; the non-empty rows in order in S.de
      const uint4 row = lane < 9 ? S.row[9 * s + lane] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t start = row.x, cnt = row.y;
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const uint32_t v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
      }
      const uint32_t at = incl - cnt - 32u * static_cast<unsigned>(turn0);  // less the turns before
      const unsigned some = __ballot_sync(full, cnt > 0);
      if (cnt) S.de[__popc(some & upto) - 1] = make_int2(static_cast<int>(start - at), static_cast<int>(row.z));
      // the 8 slots of the group's eighth, in pairs
      const bool whole = (f & 7) == 0 && l == f + 7;
      const uint32_t ta = static_cast<uint32_t>(__cvta_generic_to_shared(&S.txy[(f & ~7) >> 1]));
      const uint32_t tb = static_cast<uint32_t>(__cvta_generic_to_shared(&S.tz[(f & ~7) >> 1]));
      __syncwarp();
      // non-empty rows begun before the turn, less one
      int rows = __popc(__ballot_sync(full, cnt > 0 && static_cast<int>(at) < 0)) - 1;
      for (int c = 0; 32 * c < T; ++c) {
        const int k = 32 * c + lane;
        const unsigned rel = at - 32u * static_cast<unsigned>(c);
        const unsigned begun = __reduce_or_sync(full, (cnt && rel < 32u) ? 1u << rel : 0u);  // rows that begin here
        float4 xj;
        xj.x = NAN;  // no candidate: no hit, also for an h2 beyond FP32's range (infinity)
        if (k < T) {
          const int2 de = S.de[rows + __popc(begun & upto)];
          const int j = k + de.x;
          xj = ld<NC>(&xs[j]);
          S.ent[eoff + k] = static_cast<uint16_t>(j + de.y);
        }
        rows += __popc(begun);
        const float2 X = make_float2(xj.x, xj.x), Y = make_float2(xj.y, xj.y), Z = make_float2(xj.z, xj.z);
        uint32_t m[8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float2 x, y, z;  // read each turn (broadcasts): held in registers they cost a fifth of the warps in flight
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(x.x), "=f"(x.y), "=f"(y.x), "=f"(y.y)
                       : "r"(ta + 16 * p));
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(z.x), "=f"(z.y) : "r"(tb + 8 * p));
          const float2 dx = __fadd2_rn(X, x), dy = __fadd2_rn(Y, y), dz = __fadd2_rn(Z, z);
          // each square rounded, then added as square * 1 + sum: a packed add here would be
          // contracted with the packed square into one rounding
          const float2 sq = __ffma2_rn(__fmul2_rn(dy, dy), ones, __fmul2_rn(dx, dx));
          const float2 r2 = __ffma2_rn(__fmul2_rn(dz, dz), ones, sq);
          m[2 * p] = __ballot_sync(full, r2.x <= P.h2);
          m[2 * p + 1] = __ballot_sync(full, r2.y <= P.h2);
        }
        if (whole) {
          if (lane < 2)
            *reinterpret_cast<uint4*>(&S.mask[c][f + 4 * lane]) =
                lane ? make_uint4(m[4], m[5], m[6], m[7]) : make_uint4(m[0], m[1], m[2], m[3]);
        } else if (lane >= f && lane <= l) {  // the eighth holds slots of other groups too
          uint32_t own = m[0];
#pragma unroll
          for (int u = 1; u < 8; ++u) own = (lane & 7) == u ? m[u] : own;
          S.mask[c][lane] = own;
        }
      }
      __syncwarp();
      // the own slot, a hit at distance 0 in the middle row
      const uint32_t s4 = __shfl_sync(full, start, 4), a4 = __shfl_sync(full, at, 4), c4 = __shfl_sync(full, cnt, 4);
      const uint32_t own = static_cast<uint32_t>(i) - s4, k4 = a4 + own;
      if (lane >= f && lane <= l && own < c4 && k4 < static_cast<uint32_t>(T))
        S.mask[k4 >> 5][lane] &= ~(1u << (k4 & 31u));
      __syncwarp();
      if (PARTS && T < rest) {  // the rest of its candidates in the rounds after
        turn0 += kNbrWords;
        break;
      }
      turn0 = 0;
    }
    // lists: the lanes take their hits in order, each the next set bit of its words (words
    // without a hit are skipped by the mask of the others), all at the same entry index
    int total = 0, have = 0;
    unsigned words_left = 0;
    const bool mine = live && group >= s_begin && group < s + (turn0 ? 1 : 0);
    int own_at = 0;
    if (mine) {
      own_at = S.eoff[group];
      const int skip = group == s_begin ? t_begin : 0;
      const int nw = min((S.cand[group] - 32 * skip + 31) >> 5, kNbrWords);
      if (skip) have = nbr_total(hdr[i]);
      for (int c = 0; c < nw; ++c) {
        const uint32_t m = S.mask[c][lane];
        total += __popc(m);
        words_left |= m ? 1u << c : 0u;
      }
    }
    const int room = P.max_words * 2 - have;
    if (total > room) {
      atomicOr(err, PBF_ERRBIT_NEIGHBOR_CAPACITY);
      total = room;
    }
    if (mine) {
      const uint32_t g0 = S.gb[3 * group];
      // the slab bases relative to slab 0's, less the tag bits (nbr_decode)
      hdr[i] = make_uint4(g0, S.gb[3 * group + 1] - g0 - (1u << kOffsetBits),
                          S.gb[3 * group + 2] - g0 - (2u << kOffsetBits), static_cast<uint32_t>(have + total));
    }
    const int most = __reduce_max_sync(full, total);
    uint4* out = reinterpret_cast<uint4*>(words) + i;
    uint32_t m = 0;
    const uint16_t* ent = S.ent + own_at;
    for (int k = 0; k < most; k += 8) {
      uint32_t q[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (m == 0) {  // past its last hit a lane rereads word 0: what it collects there is not stored or not counted
          const int w = max(__ffs(words_left) - 1, 0);
          words_left &= words_left - 1;
          m = S.mask[w][lane];
          ent = S.ent + own_at + 32 * w;
        }
        q[u] = ent[(__ffs(m) - 1) & 31];
        m &= m - 1;
      }
      if (!PARTS || t_begin == 0) {
        if (k < total)
          out[static_cast<size_t>(k >> 3) * n] =
              make_uint4(q[0] | q[1] << 16, q[2] | q[3] << 16, q[4] | q[5] << 16, q[6] | q[7] << 16);
      } else {  // behind the entries of the pieces before
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int e = have + k + u;
          if (k + u < total)
            reinterpret_cast<uint16_t*>(out + static_cast<size_t>(e >> 3) * n)[e & 7] = static_cast<uint16_t>(q[u]);
        }
      }
    }
    __syncwarp();
  } while (s < ng);
  return kNbrDone;
}

// Builds the list of slot i (lane's slot of a warp of 32 consecutive ones; i >= n: none). S: the
// warp's shared tables. one: 1, unknown to the compiler. DENSE: groups beyond the words in pieces
// (false: by the thread scan, for a kernel that has no room for the code).
template <bool NC, bool DENSE>
__device__ __forceinline__ void nbr_build_warp(NbrWarp& S, int i, const float4* xs, const float4* pos,
                                               const uint32_t* cell_start, const SceneDesc* __restrict__ scenes,
                                               uint4* hdr, uint32_t* words, unsigned* err, const DevParams& P,
                                               float one, int n) {
  NbrResult r = nbr_build_lists<NC, false>(S, i, xs, pos, cell_start, scenes, hdr, words, err, P, one, n);
  if (r == kNbrDone) return;
  if (DENSE && r == kNbrParts)
    nbr_build_lists<NC, true>(S, i, xs, pos, cell_start, scenes, hdr, words, err, P, one, n);
  else if (i < n)
    nbr_scan_thread<NC>(i, xs, pos, cell_start, scenes, hdr, words, err, P, n);
}

}  // namespace pbf
