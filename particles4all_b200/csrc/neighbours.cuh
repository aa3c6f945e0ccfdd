// neighbours.cuh — the neighbour walk shared by the gather passes.
//
// The reference walks, for particle i, the 3x3 row ranges
// [cellStart[row+x0], cellStart[row+x1+1]) of the cell block around
// cellOf(pred_i) and tests every candidate j against r^2 < h^2 (src/wgsl.js:98-111),
// the boundary samples of a row after its fluid particles (src/wgsl.js:497-533).
// Here that walk is split in two phases:
//   1. build_list tests every candidate once and appends the ones within a radius
//      (h, or h + skin for lists that later Jacobi iterations reuse) to the
//      particle's neighbour list, in the reference's visiting order: rows z->y,
//      fluid j ascending, then the row's boundary samples (tagged kBoundTag);
//   2. walk2 / walk2g run the pass's real work over the list, two entries per loop
//      iteration (pair_math.cuh), every entry re-tested against r^2 < h^2 with the
//      current positions by the pass itself, the sums taken in list order.
// Phase 2 therefore visits exactly the reference's neighbours in exactly its
// order, so sums are bit-identical, while the expensive in-range work no longer
// runs warp-wide on every candidate, and the loop has no per-row bookkeeping:
// lanes of a warp hold different numbers of neighbours per row, so a walk that
// switches rows inside the loop pays the switch in almost every iteration.
// The list is stored [entry / 2][particle][2] (list_at), so the lanes of a warp read
// two entries of 32 consecutive particles with one coalesced 8-byte load. The
// particle itself is never listed (it contributes to no pass), except that a list of
// odd length is padded with it: r^2 = 0 contributes to no pass but lambda's density,
// which tests for it. A particle with more than kListCap entries is marked
// kListOverflow and walked with the reference's direct loop instead.
#pragma once
#include "p4a_math.cuh"
#include "pair_math.cuh"

namespace p4a {

constexpr int kRows = 9;
constexpr uint32_t kListOverflow = 0xffffffffu;  // count of a particle whose list did not fit
constexpr uint32_t kBoundTag = 0x80000000u;      // entry = kBoundTag | boundary sample index
constexpr uint32_t kHasBound = 0x40000000u;      // count flag: the list holds boundary samples
constexpr uint32_t kCountMask = 0x0000ffffu;
constexpr int kBuildShift = 16;                  // count bits 16-19: the iteration that built the list

// Place of entry k of particle i in a list array of `cap` particles.
__device__ __forceinline__ size_t list_at(uint32_t k, uint32_t cap, uint32_t i) {
  return 2 * ((size_t)(k >> 1) * cap + i) + (k & 1u);
}

// Row r = 3*(dz+1) + (dy+1), the reference's dz-outer, dy-inner order.
struct RowWalk {
  int x0, x1;
  I3 c;
  __device__ __forceinline__ RowWalk(const SimParams& P, F3 p) {
    c = cell_of(P, p);
    x0 = max(c.x - 1, 0);
    x1 = min(c.x + 1, P.gridDim[0] - 1);
  }
  // Row base index of row r, or -1 when the row is outside the grid.
  __device__ __forceinline__ int row_base(const SimParams& P, int r) const {
    const int z = c.z + r / 3 - 1, y = c.y + r % 3 - 1;
    if (z < 0 || z >= P.gridDim[2] || y < 0 || y >= P.gridDim[1]) return -1;
    return (z * P.gridDim[1] + y) * P.gridDim[0];
  }
};

// Bit k: point k of pts[0, n), n <= 32, lies within r^2 < r2lim of p. Reads whole groups
// of four points: position arrays have kReadPad elements more than they hold particles.
__device__ __forceinline__ uint32_t near_bits(F3 p, const float4* __restrict__ pts, uint32_t n, float r2lim) {
  uint32_t m = 0u;
#pragma unroll 1
  for (uint32_t k = 0; k < n; k += 4u) {
    const float4 q0 = __ldg(&pts[k]), q1 = __ldg(&pts[k + 1]), q2 = __ldg(&pts[k + 2]), q3 = __ldg(&pts[k + 3]);
    const F3 d0 = sub3(p, xyz(q0)), d1 = sub3(p, xyz(q1)), d2 = sub3(p, xyz(q2)), d3 = sub3(p, xyz(q3));
    uint32_t g = dot3(d0, d0) < r2lim ? 1u : 0u;
    if (dot3(d1, d1) < r2lim) g |= 2u;
    if (dot3(d2, d2) < r2lim) g |= 4u;
    if (dot3(d3, d3) < r2lim) g |= 8u;
    m |= g << k;
  }
  return m & (0xffffffffu >> (32u - n));
}

// Phase 1: the list of particle i (scene-local cellStart cs / bcs, arena index i)
// with every candidate j != i of the nine rows within r^2 < r2lim, and, when B,
// every boundary sample of each row within r^2 < r2lim after the row's fluid
// candidates. Returns the entry count (| kHasBound when boundary samples were
// listed), or kListOverflow.
// A row's candidates are tested first, into a bit mask, and only the ones within the
// radius are then appended: of the 27 cells' 216 candidates about 35 are, and some lane of
// a warp has one at nearly every candidate, so appending as they are tested runs the
// append 216 times. What is left is bound by the loads of the candidates: 16 bytes for
// each lane, four cycles of the L1 each (88 % busy). us per launch of lambda, a list built
// in every launch (preset, 62,742) 68.9 -> 48.2, in the first of a substep's (one scene of
// 32,768 / 264k / 2.1M) 28.1 -> 26.3 / 56.4 -> 55.5 / 284 -> 276, 96 mixed scenes
// 539 -> 492; xsph with a list of its own (preset) 74.5 -> 59.7.
template <bool B>
__device__ __forceinline__ uint32_t build_list(const SimParams& P, const RowWalk& w, uint32_t i, F3 pi,
                                               const float4* __restrict__ pred,
                                               const uint32_t* __restrict__ cs,
                                               const uint32_t* __restrict__ bcs,
                                               const float4* __restrict__ bpos, uint32_t* __restrict__ list,
                                               uint32_t cap, float r2lim) {
  uint32_t c = 0, flags = 0u, held = 0u;
  // entries are stored two at a time: `held` is the first of a pair
  uint2* __restrict__ out = reinterpret_cast<uint2*>(list) + i;
  // appends the points of [b, e) within the radius, 32 candidates at a time
  auto row = [&](const float4* __restrict__ pts, uint32_t b, uint32_t e, uint32_t tag) {
#pragma unroll 1
    for (uint32_t base = b; base < e; base += 32u) {
      const uint32_t n = min(e - base, 32u);
      uint32_t m = near_bits(pi, pts + base, n, r2lim);
      if (tag == 0u && i - base < 32u) m &= ~(1u << (i - base));
      if (c + (uint32_t)__popc(m) > kListCap) {  // overflow: the list is not used
        c = kListCap + 1u;
        m = 0u;
      }
      if (tag != 0u && m != 0u) flags = kHasBound;
      for (; m != 0u; m &= m - 1u) {
        const uint32_t at = tag | (base + (uint32_t)__ffs((int)m) - 1u);
        if ((c & 1u) != 0u) {
          *out = make_uint2(held, at);
          out += cap;
        }
        held = at;
        c++;
      }
    }
  };
#pragma unroll 1
  for (int r = 0; r < kRows; r++) {
    const int rb = w.row_base(P, r);
    if (rb < 0) continue;
    row(pred, __ldg(&cs[rb + w.x0]), min(__ldg(&cs[rb + w.x1 + 1]), P.pEnd), 0u);
    if constexpr (B) {
      if (P.nBoundary > 0u) row(bpos, __ldg(&bcs[rb + w.x0]), __ldg(&bcs[rb + w.x1 + 1]), kBoundTag);
    }
  }
  if ((c & 1u) != 0u && c < kListCap) *out = make_uint2(held, i);
  return c > kListCap ? kListOverflow : c | flags;
}

// build_list for one particle (iL, piL, its row walk wL) by all 32 lanes of a warp:
// lane k tests candidate base + k of each row, and a ballot orders the appends, so
// the list (entries, order, count, flags) is the one build_list writes.
template <bool B>
__device__ __forceinline__ uint32_t build_list_coop(const SimParams& P, const RowWalk& wL, uint32_t iL, F3 piL,
                                                    const float4* __restrict__ pred,
                                                    const uint32_t* __restrict__ cs,
                                                    const uint32_t* __restrict__ bcs,
                                                    const float4* __restrict__ bpos, uint32_t* __restrict__ list,
                                                    uint32_t cap, float r2lim) {
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  uint32_t c = 0, flags = 0u;
#pragma unroll 1
  for (int r = 0; r < kRows; r++) {
    const int rb = wL.row_base(P, r);
    if (rb < 0) continue;
    const uint32_t b = __ldg(&cs[rb + wL.x0]);
    const uint32_t e = min(__ldg(&cs[rb + wL.x1 + 1]), P.pEnd);
    for (uint32_t base = b; base < e; base += 32u) {
      const uint32_t j = base + lane;
      bool in = false;
      if (j < e && j != iL) {
        const F3 dd = sub3(piL, xyz(__ldg(&pred[j])));
        in = dot3(dd, dd) < r2lim;
      }
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const uint32_t pos = c + (uint32_t)__popc(m & below);
        if (pos < kListCap) list[list_at(pos, cap, iL)] = j;
      }
      c += (uint32_t)__popc(m);
    }
    if constexpr (B) {
      if (P.nBoundary > 0u) {
        const uint32_t bb = __ldg(&bcs[rb + wL.x0]), be = __ldg(&bcs[rb + wL.x1 + 1]);
        for (uint32_t base = bb; base < be; base += 32u) {
          const uint32_t k = base + lane;
          bool in = false;
          if (k < be) {
            const F3 dd = sub3(piL, xyz(__ldg(&bpos[k])));
            in = dot3(dd, dd) < r2lim;
          }
          const uint32_t m = __ballot_sync(0xffffffffu, in);
          if (in) {
            const uint32_t pos = c + (uint32_t)__popc(m & below);
            if (pos < kListCap) list[list_at(pos, cap, iL)] = kBoundTag | k;
          }
          if (m) flags = kHasBound;
          c += (uint32_t)__popc(m);
        }
      }
    }
  }
  if ((c & 1u) != 0u && c < kListCap && lane == 0u) list[list_at(c, cap, iL)] = iL;
  return c > kListCap ? kListOverflow : c | flags;
}

// The lanes of a warp that `need` a new list get one; all 32 lanes must call.
// When few lanes need one, the whole warp builds each of their lists in turn
// (build_list_coop), instead of letting the warp wait while those lanes test
// their ~216 candidates one by one; when many do, each lane builds its own.
// Returns the lane's new count word, or `current` for lanes that need none.
constexpr int kCoopLanes = 2;
template <bool B>
__device__ __forceinline__ uint32_t build_lists_warp(const SimParams& P, bool need, const RowWalk& w, uint32_t i,
                                                     F3 pi, const float4* __restrict__ pred,
                                                     const uint32_t* __restrict__ cs,
                                                     const uint32_t* __restrict__ bcs,
                                                     const float4* __restrict__ bpos, uint32_t* __restrict__ list,
                                                     uint32_t cap, float r2lim, uint32_t current) {
  const unsigned needMask = __ballot_sync(0xffffffffu, need);
  if (needMask == 0u) return current;
  if (__popc(needMask) > kCoopLanes) return need ? build_list<B>(P, w, i, pi, pred, cs, bcs, bpos, list, cap, r2lim)
                                                 : current;
  const int lane = (int)(threadIdx.x & 31u);
  uint32_t out = current;
  for (unsigned m = needMask; m != 0u; m &= m - 1u) {
    const int L = __ffs(m) - 1;
    RowWalk wL = w;
    wL.c.x = __shfl_sync(0xffffffffu, w.c.x, L);
    wL.c.y = __shfl_sync(0xffffffffu, w.c.y, L);
    wL.c.z = __shfl_sync(0xffffffffu, w.c.z, L);
    wL.x0 = __shfl_sync(0xffffffffu, w.x0, L);
    wL.x1 = __shfl_sync(0xffffffffu, w.x1, L);
    const uint32_t iL = __shfl_sync(0xffffffffu, i, L);
    const F3 piL = {__shfl_sync(0xffffffffu, pi.x, L), __shfl_sync(0xffffffffu, pi.y, L),
                    __shfl_sync(0xffffffffu, pi.z, L)};
    const uint32_t cnt = build_list_coop<B>(P, wL, iL, piL, pred, cs, bcs, bpos, list, cap, r2lim);
    if (lane == L) out = cnt;
  }
  return out;
}

// Whether particle i, now in `cell`, may walk its stored list before iteration `it`
// of this substep (it = iters: the positions after the last iteration). The list
// was built at iteration b (its count word's bits 16-19) from the positions then,
// with radius h + skin, in the cell recorded in nbCell. It still holds every pair
// now within h when the particle is in the same cell (same candidate rows) and
// every candidate (the particles sorted into the block's cells) and the particle
// itself moved at most skin / 2 since iteration b, by either bound:
//  - S: the sum of the iterations' largest single-iteration displacements since b
//    over the whole scene (disp[t], recorded by every delta and rigid projection);
//  - V: per block cell, the largest displacement of the cell's particles from the
//    substep's start positions now, plus the same at iteration b (cellDisp[t] after
//    iteration t), since |p(now) - p(b)| <= |p(now) - ref| + |p(b) - ref|.
// V is local: a fast particle elsewhere in the scene does not force this list to
// be rebuilt.
__device__ __forceinline__ bool list_reusable(const SimParams& P, const DevScene& d, int it, uint32_t i,
                                              const RowWalk& w, uint32_t cell, uint32_t countWord) {
  if (it <= 0 || it >= kDispSlots || countWord == kListOverflow) return false;
  if (__ldg(&d.nbCell[i]) != cell) return false;
  const int b = (int)((countWord >> kBuildShift) & 0xfu);
  if (b >= it) return false;
  const float* disp = d.disp + (size_t)P.slot * kDispSlots;
  float S = 0.0f;
  for (int t = b; t < it; t++) S += __ldg(&disp[t]);
  if (S * 1.00001f <= P.skinHalf) return true;
  const float* vNow = d.cellDisp + (size_t)(it - 1) * d.cellStride + P.cOff;
  const float* vB = b > 0 ? d.cellDisp + (size_t)(b - 1) * d.cellStride + P.cOff : nullptr;
  // the particle's own sort cell (the cell of its start position) may lie outside
  // the block when it moved more than a cell since the sort
  const I3 a = cell_of(P, xyz(__ldg(&d.nbRef[i])));
  const uint32_t ac = cell_index(P, a);
  float V = __ldg(&vNow[ac]) + (vB ? __ldg(&vB[ac]) : 0.0f);
  // The 27 cells with every load independent of the others (a loop over rows with
  // a data-dependent skip issued them row by row, one memory latency per row): a
  // row outside the grid reads the particle's own row and counts as 0, and x is
  // clamped into the grid, which repeats x0 or x1 at an edge. The slots hold
  // displacement lengths, so neither changes the maximum.
  const int gx = P.gridDim[0], gy = P.gridDim[1], gz = P.gridDim[2];
  const int ownRow = (w.c.z * gy + w.c.y) * gx;
#pragma unroll
  for (int r = 0; r < kRows; r++) {
    const int z = w.c.z + r / 3 - 1, y = w.c.y + r % 3 - 1;
    const bool in = z >= 0 && z < gz && y >= 0 && y < gy;
    const int rb = in ? (z * gy + y) * gx : ownRow;
#pragma unroll
    for (int dx = -1; dx <= 1; dx++) {
      const int x = min(max(w.c.x + dx, 0), gx - 1);
      const float v = __ldg(&vNow[rb + x]) + (vB ? __ldg(&vB[rb + x]) : 0.0f);
      V = fmaxf(V, in ? v : 0.0f);
    }
  }
  return V * 1.00001f <= P.skinHalf;
}

// Phase 2: pair(e, q0, q1) for every two entries e.x, e.y of the list (e.y is the
// particle itself when the count is odd and this is the last pair), with q0, q1 =
// fsrc[entry] of a fluid entry and, when B, bsrc[sample] of a boundary entry (e still
// carries its tag). Without B the list holds no boundary samples. The loop is software
// pipelined: while a pair is processed, the next pair's gathers and the list load after
// it are in flight, so the latency of the dependent list-then-gather chain overlaps
// the arithmetic.
// With FAR the pair four ahead is prefetched into the L2: see far_lists.
template <bool B, bool FAR, class FPair>
__device__ __forceinline__ void walk2(const uint32_t* list, uint32_t cap, uint32_t i, uint32_t count,
                                      const float4* __restrict__ fsrc, const float4* __restrict__ bsrc,
                                      FPair&& pair) {
  const uint32_t pairs = ((count & kCountMask) + 1u) >> 1;
  if (pairs == 0u) return;
  auto fetch = [&](uint32_t e) {
    if constexpr (B) return __ldg(((e & kBoundTag) != 0u ? bsrc : fsrc) + (e & ~kBoundTag));
    return __ldg(fsrc + e);
  };
  // plain loads: the same kernel may have just written the list
  const uint2* at = reinterpret_cast<const uint2*>(list) + i;
  uint2 e = *at, en = e;
  float4 q0 = fetch(e.x), q1 = fetch(e.y);
  if (pairs > 1u) {
    at += cap;
    en = *at;
  }
  for (uint32_t k = 1u; k <= pairs; k++) {
    const uint2 ec = e;
    const float4 c0 = q0, c1 = q1;
    if (k < pairs) {
      e = en;
      q0 = fetch(e.x);
      q1 = fetch(e.y);
      if (k + 1u < pairs) {
        at += cap;
        en = *at;
        if (FAR && k + 4u < pairs) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 3 * (size_t)cap));
      }
    }
    pair(ec, c0, c1);
  }
}

// The reference's direct loop (particles whose list overflowed): every candidate
// j != self of the nine rows with r^2 < h^2 (the particle itself contributes to
// no pass), then, when B, the row's boundary samples with 1e-12 <= r^2 < h^2. fsrc
// holds the candidate positions in .xyz (and whatever the pass keeps in .w).
template <bool B, class FFluid, class FBound>
__device__ __forceinline__ void walk_direct(const SimParams& P, const RowWalk& w, F3 pi, uint32_t self,
                                            const float4* __restrict__ fsrc, const uint32_t* __restrict__ cs,
                                            const uint32_t* __restrict__ bcs, const float4* __restrict__ bpos,
                                            FFluid&& fluid, FBound&& bound) {
#pragma unroll 1
  for (int r = 0; r < kRows; r++) {
    const int rb = w.row_base(P, r);
    if (rb < 0) continue;
    const uint32_t b = __ldg(&cs[rb + w.x0]);
    const uint32_t e = min(__ldg(&cs[rb + w.x1 + 1]), P.pEnd);
    for (uint32_t j = b; j < e; j++) {
      const float4 q = __ldg(&fsrc[j]);
      const F3 d = sub3(pi, xyz(q));
      if (dot3(d, d) < P.h2 && j != self) fluid(j, q);
    }
    if constexpr (B) {
      if (P.nBoundary > 0u) {
        const uint32_t bb = __ldg(&bcs[rb + w.x0]), be = __ldg(&bcs[rb + w.x1 + 1]);
        for (uint32_t k = bb; k < be; k++) {
          const float4 q = __ldg(&bpos[k]);
          const F3 d = sub3(pi, xyz(q));
          const float r2 = dot3(d, d);
          if (r2 < P.h2 && r2 >= 1.0e-12f) bound(k, q);
        }
      }
    }
  }
}

// The walk of the fluid-only passes (xsph, normals, tension): pair(j0, j1, q0, q1, g0,
// g1) for every two entries, q = pred[j] and g = gsrc[j] (the pass's packed
// per-neighbour values), both gathered in the pipeline. A boundary entry of a reused
// list is replaced by the particle itself, as the padding is: j == i is skipped by the
// pass.
template <class FPair>
__device__ __forceinline__ void walk2g(const uint32_t* list, uint32_t cap, uint32_t i, uint32_t count,
                                       const float4* __restrict__ pred, const float4* __restrict__ gsrc,
                                       FPair&& pair) {
  const uint32_t pairs = ((count & kCountMask) + 1u) >> 1;
  if (pairs == 0u) return;
  auto slot = [&](uint32_t e) { return (e & kBoundTag) != 0u ? i : e; };
  const uint2* at = reinterpret_cast<const uint2*>(list) + i;
  uint2 e = *at;
  uint32_t j0 = slot(e.x), j1 = slot(e.y);
  float4 q0 = __ldg(pred + j0), q1 = __ldg(pred + j1), g0 = __ldg(gsrc + j0), g1 = __ldg(gsrc + j1);
  if (pairs > 1u) {
    at += cap;
    e = *at;
  }
  for (uint32_t k = 1u; k <= pairs; k++) {
    const uint32_t i0 = j0, i1 = j1;
    const float4 c0 = q0, c1 = q1, h0 = g0, h1 = g1;
    if (k < pairs) {
      j0 = slot(e.x);
      j1 = slot(e.y);
      q0 = __ldg(pred + j0);
      q1 = __ldg(pred + j1);
      g0 = __ldg(gsrc + j0);
      g1 = __ldg(gsrc + j1);
      if (k + 1u < pairs) {
        at += cap;
        e = *at;
      }
    }
    pair(i0, i1, c0, c1, h0, h1);
  }
}

// The fluid-only passes with the IEEE operations: visit(pred[j], gsrc[j]) of every listed
// fluid entry, or of the reference's direct loop for an overflowed list.
template <class F>
__device__ __forceinline__ void walk_fluid(const SimParams& P, const RowWalk& w, uint32_t i, F3 pi,
                                           const float4* __restrict__ pred, const float4* __restrict__ gsrc,
                                           const uint32_t* __restrict__ cs, const uint32_t* __restrict__ list,
                                           uint32_t cap, uint32_t count, F&& visit) {
  if (count == kListOverflow) {
    walk_direct<false>(P, w, pi, i, pred, cs, nullptr, nullptr,
                       [&](uint32_t j, float4 q) { visit(q, __ldg(&gsrc[j])); }, [](uint32_t, float4) {});
    return;
  }
  walk2g(list, cap, i, count, pred, gsrc, [&](uint32_t j0, uint32_t j1, float4 q0, float4 q1, float4 g0, float4 g1) {
    if (j0 != i) visit(q0, g0);
    if (j1 != i) visit(q1, g1);
  });
}

}  // namespace p4a
