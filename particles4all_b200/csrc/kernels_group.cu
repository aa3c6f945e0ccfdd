// kernels_group.cu — the neighbour passes of small plain scenes with a group of G lanes
// per particle.
//
// One thread per particle leaves most of the GPU idle in a small scene (2,197 particles
// are 69 warps on 148 SMs), and each pass then takes as long as one thread needs for its
// chain of dependent loads: 216 candidates tested four at a time, then 35 list entries.
// Here the G lanes of a group test G candidates at a time (a ballot orders the appends:
// the lists are the ones build_list writes), and form the pair terms of G entries at a
// time. The sums keep the reference's order: the terms of 32
// entries go to shared memory, and one lane per component adds them up entry after entry
// with the fused multiply-add that the sum is defined by, acc = fma(a, b, acc) (a plain
// addition is fma(1, b, acc); an entry that does not contribute has a zero term, which
// leaves every sum as it is). Roots and quotients are those of pair_math.cuh (FAST), or
// the IEEE operations for parameters outside its ranges. Bound by the latency of those
// chains, whose length falls with G; a frame of 2,197 particles takes 167 us with 16 lanes
// and 262 us with one thread per particle (group_lanes in api.cu has the other sizes).
// 32 lanes gain 3 % more below 3,000 particles and lose above: not built.
#include <cuda_runtime.h>

#include "neighbours.cuh"
#include "p4a_internal.h"
#include "p4a_math.cuh"

namespace p4a {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kTB = 128;
// Entries whose terms are in shared memory at a time: five of each lane of a group of 8,
// which most lists fit. Rows are padded so that the lanes that sum, four entries per
// 16-byte load, read different banks.
template <int G>
constexpr int kChunk = G == 8 ? 40 : 32;
template <int G>
constexpr int kRow = kChunk<G> + 4;

// The root of r^2 with the quotients by it, and quotients by a density.
struct Root {
  float s, yn;
};
template <bool FAST>
__device__ __forceinline__ Root root_of(float x) {
  if constexpr (FAST) {
    const Root1 r = root1(x);
    return {r.s, r.yn};
  }
  return {sqrtf(x), 0.0f};
}
template <bool FAST>
__device__ __forceinline__ float over(float a, Root r) {
  if constexpr (FAST) return quot1(a, r.s, r.yn);
  return a / r.s;
}
template <bool FAST>
__device__ __forceinline__ Root density_of(float d) {
  if constexpr (FAST) return {d, recip1(d)};
  return {d, 0.0f};
}

// A warp's lanes in groups of G.
template <int G>
struct Group {
  int lane, sub, first;     // lane of the warp, lane of the group, the group's first lane
  uint32_t members, below;  // the group's lanes, and those before this one
  __device__ __forceinline__ Group() {
    lane = (int)threadIdx.x & 31;
    sub = lane & (G - 1);
    first = lane - sub;
    members = ((1u << G) - 1u) << first;
    below = members & ((1u << lane) - 1u);
  }
  template <class T>
  __device__ __forceinline__ T from(T v, int s) const { return __shfl_sync(kFull, v, first + s); }
  __device__ __forceinline__ float max_all(float v) const {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
  }
};

// list_reusable (neighbours.cuh) by a group: the 27 cells shared among its lanes. All
// lanes of the warp call; `act` groups get the answer, the others false.
template <int G>
__device__ __forceinline__ bool group_reusable(const Group<G>& g, const SimParams& P, const DevScene& d, int it,
                                               uint32_t i, const RowWalk& w, uint32_t cell, uint32_t countWord,
                                               bool act) {
  const int b = (int)((countWord >> kBuildShift) & 0xfu);
  const bool may = act && it > 0 && it < kDispSlots && countWord != kListOverflow && b < it &&
                   __ldg(&d.nbCell[i]) == cell;
  const float* disp = d.disp + (size_t)P.slot * kDispSlots;
  float S = 0.0f;
  if (may)
    for (int t = b; t < it; t++) S += __ldg(&disp[t]);
  const bool whole = may && S * 1.00001f <= P.skinHalf;
  const bool local = may && !whole;
  float V = 0.0f;
  if (local) {
    const float* vNow = d.cellDisp + (size_t)(it - 1) * d.cellStride + P.cOff;
    const float* vB = b > 0 ? d.cellDisp + (size_t)(b - 1) * d.cellStride + P.cOff : nullptr;
    const uint32_t ac = cell_index(P, cell_of(P, xyz(__ldg(&d.nbRef[i]))));
    V = __ldg(&vNow[ac]) + (vB ? __ldg(&vB[ac]) : 0.0f);
    for (int t = g.sub; t < 27; t += G) {
      const int z = w.c.z + t / 9 - 1, y = w.c.y + t / 3 % 3 - 1;
      if (z < 0 || z >= P.gridDim[2] || y < 0 || y >= P.gridDim[1]) continue;
      const int x = min(max(w.c.x + t % 3 - 1, 0), P.gridDim[0] - 1);
      const int at = (z * P.gridDim[1] + y) * P.gridDim[0] + x;
      V = fmaxf(V, __ldg(&vNow[at]) + (vB ? __ldg(&vB[at]) : 0.0f));
    }
  }
  V = g.max_all(V);
  return whole || (local && V * 1.00001f <= P.skinHalf);
}

// build_list (neighbours.cuh) by a group: G candidates are tested at a time and a ballot
// orders the appends, so the list (entries, order, count, flags) is the one build_list
// writes. The bounds of the nine rows come in one round of loads and a row's candidates
// in another. The list is put together in shared memory (`mine`, kListCap entries) and
// stored two entries at a time, the groups of a warp side by side. All lanes of the warp
// call; groups that do not `need` a list keep `current`.
template <int G, bool B>
__device__ __forceinline__ uint32_t group_build(const Group<G>& g, const SimParams& P, bool need, const RowWalk& w,
                                                uint32_t i, F3 pi, const float4* __restrict__ pred,
                                                const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bcs,
                                                const float4* __restrict__ bsample, uint32_t* mine, uint32_t* list,
                                                uint32_t cap, float r2lim, uint32_t current) {
  if (!__any_sync(kFull, need)) return current;
  // lane s of the group holds the bounds of row s, all hold those of row 8
  auto bounds = [&](const uint32_t* __restrict__ starts, int r, uint32_t limit) {
    const int rb = w.row_base(P, r);
    if (!need || rb < 0) return make_uint2(0u, 0u);
    return make_uint2(__ldg(&starts[rb + w.x0]), min(__ldg(&starts[rb + w.x1 + 1]), limit));
  };
  const bool walls = B && P.nBoundary > 0u;
  const uint2 row = bounds(cs, min(g.sub, 8), P.pEnd), last = bounds(cs, 8, P.pEnd);
  uint2 rowB = make_uint2(0u, 0u), lastB = rowB;
  if (walls) {
    rowB = bounds(bcs, min(g.sub, 8), 0xffffffffu);
    lastB = bounds(bcs, 8, 0xffffffffu);
  }
  // rows whose boundary samples some group of the warp has to test
  const bool anyWall = walls && __any_sync(kFull, rowB.x < rowB.y || lastB.x < lastB.y);
  uint32_t c = 0u, flags = 0u;
  auto append = [&](bool in, uint32_t e) {
    const uint32_t m = __ballot_sync(kFull, in), pos = c + (uint32_t)__popc(m & g.below);
    if (in && pos < kListCap) mine[pos] = e;
    c += (uint32_t)__popc(m & g.members);
  };
  constexpr int U = G == 16 ? 2 : 3;  // candidates of a lane in flight
#pragma unroll 1
  for (int r = 0; r < kRows; r++) {
    const int s = r < 8 ? r : 0;
    const uint32_t fb = g.from(row.x, s), fe = g.from(row.y, s);
    const uint32_t from = r < 8 ? fb : last.x, to = r < 8 ? fe : last.y;
    for (uint32_t base = from; __any_sync(kFull, base < to); base += (uint32_t)(G * U)) {
      float4 q[U];
#pragma unroll
      for (int u = 0; u < U; u++) q[u] = __ldg(&pred[min(base + (uint32_t)(u * G + g.sub), P.pEnd - 1u)]);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const uint32_t j = base + (uint32_t)(u * G + g.sub);
        const F3 dd = sub3(pi, xyz(q[u]));
        append(j < to && dot3(dd, dd) < r2lim && j != i, j);
      }
    }
    if (anyWall) {
      const uint32_t wb = g.from(rowB.x, s), we = g.from(rowB.y, s);
      const uint32_t bFrom = r < 8 ? wb : lastB.x, bTo = r < 8 ? we : lastB.y;
      const uint32_t before = c;
      for (uint32_t base = bFrom; __any_sync(kFull, base < bTo); base += (uint32_t)G) {
        const uint32_t j = base + (uint32_t)g.sub;
        bool in = false;
        if (j < bTo) {
          const F3 dd = sub3(pi, xyz(__ldg(&bsample[j])));
          in = dot3(dd, dd) < r2lim;
        }
        append(in, kBoundTag | j);
      }
      if (c != before) flags = kHasBound;
    }
  }
  if ((c & 1u) != 0u && c < kListCap && g.sub == 0) mine[c] = i;
  __syncwarp();
  if (need) {
    const uint32_t pairs = (min(c, kListCap) + 1u) >> 1;
    uint2* out = reinterpret_cast<uint2*>(list) + i;
    for (uint32_t k = (uint32_t)g.sub; k < pairs; k += G)
      out[(size_t)k * cap] = reinterpret_cast<const uint2*>(mine)[k];
  }
  __syncwarp();
  return need ? (c > kListCap ? kListOverflow : c | flags) : current;
}

// The ordered sums over a list of `count` entries (0: the group has none; all lanes of
// the warp call). fetch(e) loads what the entry needs, term(e, loaded, out) writes its
// NT - 1 numbers (out[NT - 1] is 1), and sum s < NS is acc[s] = fma(out[a[s]], out[b[s]],
// acc[s]) over the entries in order. Lane s of the group starts from and returns sum s.
template <int G, int NT, int NS, class Loaded, class FFetch, class FTerm>
__device__ __forceinline__ float group_sums(const Group<G>& g, float (*sh)[NT][kRow<G>], const uint32_t* list,
                                            uint32_t cap, uint32_t i, uint32_t count, int a, int b, float acc,
                                            FFetch&& fetch, FTerm&& term) {
  constexpr int U = kChunk<G> / G;
  float (*t)[kRow<G>] = sh[threadIdx.x / G];
  const uint32_t longest = __reduce_max_sync(kFull, count);
  for (uint32_t c0 = 0u; c0 < longest; c0 += (uint32_t)kChunk<G>) {
    uint32_t e[U];
    Loaded q[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k = c0 + (uint32_t)(u * G + g.sub);
      e[u] = k < count ? list[list_at(k, cap, i)] : i;
    }
#pragma unroll
    for (int u = 0; u < U; u++) q[u] = fetch(e[u]);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = u * G + g.sub;
      float out[NT];
#pragma unroll
      for (int s = 0; s < NT; s++) out[s] = s == NT - 1 ? 1.0f : 0.0f;
      if (c0 + (uint32_t)k < count) term(e[u], q[u], out);
#pragma unroll
      for (int s = 0; s < NT; s++) t[s][k] = out[s];
    }
    __syncwarp();
    if (g.sub < NS) {
      const float4* __restrict__ ta = reinterpret_cast<const float4*>(t[a]);
      const float4* __restrict__ tb = reinterpret_cast<const float4*>(t[b]);
      const uint32_t n = min(longest - c0, (uint32_t)kChunk<G>);
#pragma unroll 2
      for (uint32_t k = 0; k < n; k += 4u) {  // past the list's end the terms are zero
        const float4 x = ta[k / 4u], y = tb[k / 4u];
        acc = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, acc))));
      }
    }
    __syncwarp();
  }
  return acc;
}

struct Pair4 {
  float4 q, g;
};

}  // namespace

// lambda (kernels_solve.cu) by groups.
template <int G, bool FAST>
__global__ void __launch_bounds__(kTB) k_lambda_g(const __grid_constant__ SimParams P,
                                                  const __grid_constant__ DevScene d, int it) {
  __shared__ __align__(16) float sh[kTB / G][8][kRow<G>];
  __shared__ __align__(8) uint32_t lists[kTB / G][kListCap];
  const Group<G> g;
  const uint32_t li = (blockIdx.x * kTB + threadIdx.x) / G;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ (it & 1)];
  const uint32_t* __restrict__ cs = d.cellStart + P.cOff;
  const uint32_t* __restrict__ bcs = d.bcellStart + P.cOff;
  const F3 pi = xyz(__ldg(&pred[i]));
  const RowWalk w(P, pi);
  const uint32_t cell = cell_index(P, w.c);
  if (it == 0 && act && g.sub == 0) d.nbRef[i] = make_float4(pi.x, pi.y, pi.z, 0.0f);
  uint32_t count = it > 0 && act ? d.nbCount[i] : kListOverflow;
  const bool keep = group_reusable(g, P, d, it, i, w, cell, count, act);  // every lane calls
  const bool need = act && !keep;
  count = group_build<G, true>(g, P, need, w, i, pi, pred, cs, bcs, d.bsample,
                               lists[threadIdx.x / G], d.nbList, d.cap, P.skinH2, count);
  if (need && g.sub == 0) {
    d.nbCount[i] = count != kListOverflow ? count | ((uint32_t)it << kBuildShift) : count;
    d.nbCell[i] = cell;
  }
  // sum s: density, gradient x y z, sum of squared gradients; terms: weight, kernel,
  // gradient factor, its three components, its square
  const bool listed = act && count != kListOverflow;
  const int sa = g.sub == 0 ? 0 : g.sub < 4 ? 2 : 7, sb = g.sub == 0 ? 1 : g.sub < 4 ? 2 + g.sub : 6;
  float acc = g.sub == 0 ? P.mass * poly6(P, 0.0f) : 0.0f;
  acc = group_sums<G, 8, 5, float4>(
      g, sh, d.nbList, d.cap, i, listed ? count & kCountMask : 0u, sa, sb, acc,
      [&](uint32_t e) { return __ldg((e & kBoundTag) != 0u ? d.bsample + (e & ~kBoundTag) : pred + e); },
      [&](uint32_t e, float4 q, float (&out)[8]) {
        const bool wall = (e & kBoundTag) != 0u;
        const F3 rij = sub3(pi, xyz(q));
        const float r2 = dot3(rij, rij);
        if (r2 >= P.h2 || (wall && r2 < 1.0e-12f)) return;
        const float t = P.h2 - r2;
        out[0] = wall ? q.w : P.mass;
        out[1] = P.poly6 * t * t * t;
        if (!wall && !(r2 > 1.0e-12f)) return;
        const Root rr = root_of<FAST>(r2);
        const float hr = P.h - rr.s;
        const float s = over<FAST>((wall ? q.w * P.invRho0 * P.spikyGrad : P.volSpiky) * hr * hr, rr);
        const F3 gr = mul3(rij, s);
        out[2] = wall ? s : 1.0f;
        out[3] = wall ? rij.x : gr.x;
        out[4] = wall ? rij.y : gr.y;
        out[5] = wall ? rij.z : gr.z;
        out[6] = wall ? 0.0f : dot3(gr, gr);
      });
  float rho = g.from(acc, 0), sumGrad2 = g.from(acc, 4);
  F3 gradSum = {g.from(acc, 1), g.from(acc, 2), g.from(acc, 3)};
  if (!act || g.sub != 0) return;
  if (!listed)
    walk_direct<true>(
        P, w, pi, i, pred, cs, bcs, d.bsample,
        [&](uint32_t, float4 q) {
          const F3 rij = sub3(pi, xyz(q));
          const float r2 = dot3(rij, rij);
          const float t = P.h2 - r2;
          rho = fmaf(P.mass, P.poly6 * t * t * t, rho);
          if (r2 > 1.0e-12f) {
            const float rr = sqrtf(r2);
            const float hr = P.h - rr;
            const F3 gr = mul3(rij, P.volSpiky * hr * hr / rr);
            gradSum = add3(gradSum, gr);
            sumGrad2 = sumGrad2 + dot3(gr, gr);
          }
        },
        [&](uint32_t, float4 q) {
          const F3 rij = sub3(pi, xyz(q));
          const float r2 = dot3(rij, rij);
          const float t = P.h2 - r2;
          rho = fmaf(q.w, P.poly6 * t * t * t, rho);
          const float rr = sqrtf(r2);
          const float hr = P.h - rr;
          gradSum = fma3(q.w * P.invRho0 * P.spikyGrad * hr * hr / rr, rij, gradSum);
        });
  d.density[i] = rho;
  const float C = rho * P.invRho0 - 1.0f;
  float lam = 0.0f;
  if (C > 0.0f) lam = -C / (dot3(gradSum, gradSum) + sumGrad2 + P.cfmEps + 1.0e-12f);
  d.lambda[i] = lam;
  d.predLam[i] = make_float4(pi.x, pi.y, pi.z, lam);
}

// delta (kernels_solve.cu) by groups.
template <int G, bool FAST>
__global__ void __launch_bounds__(kTB) k_delta_g(const __grid_constant__ SimParams P,
                                                 const __grid_constant__ DevScene d, int it) {
  __shared__ __align__(16) float sh[kTB / G][7][kRow<G>];
  const Group<G> g;
  const uint32_t li = (blockIdx.x * kTB + threadIdx.x) / G;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pl = d.predLam;
  const float4 self = __ldg(&pl[i]);
  const F3 pi = xyz(self);
  const uint32_t count = act ? __ldg(&d.nbCount[i]) : 0u;
  const bool listed = act && count != kListOverflow;
  // sums: fluid x y z, walls x y z (and, in lane 6, the fluid neighbours); terms: the
  // fluid and the wall factor, the difference, 1 for a fluid neighbour
  const int sa = g.sub < 3 ? 0 : g.sub < 6 ? 1 : 6, sb = g.sub < 6 ? 2 + g.sub % 3 : 5;
  auto grad = [&](float r2) {
    const Root rr = root_of<FAST>(r2);
    const float hr = P.h - rr.s;
    return over<FAST>(P.spikyGrad * hr * hr, rr);
  };
  auto fluid = [&](float r2, float lam) {
    const float t = P.h2 - r2;
    const float ratio = P.poly6 * t * t * t * P.sCorrWq;
    const float r2r = ratio * ratio;
    const float sc = -P.sCorrK * r2r * r2r;
    return (self.w + lam + sc) * grad(r2);
  };
  const float acc = group_sums<G, 7, 7, float4>(
      g, sh, d.nbList, d.cap, i, listed ? count & kCountMask : 0u, sa, sb, g.sub == 6 ? 1.0f : 0.0f,
      [&](uint32_t e) { return __ldg((e & kBoundTag) != 0u ? d.bsample + (e & ~kBoundTag) : pl + e); },
      [&](uint32_t e, float4 q, float (&out)[7]) {
        const F3 rij = sub3(pi, xyz(q));
        const float r2 = dot3(rij, rij);
        if (r2 >= P.h2 || r2 < 1.0e-12f) return;
        if ((e & kBoundTag) != 0u) {
          out[1] = (self.w * q.w) * grad(r2);
        } else {
          out[0] = fluid(r2, q.w);
          out[5] = 1.0f;
        }
        out[2] = rij.x;
        out[3] = rij.y;
        out[4] = rij.z;
      });
  F3 dsum = {g.from(acc, 0), g.from(acc, 1), g.from(acc, 2)}, dB = {g.from(acc, 3), g.from(acc, 4), g.from(acc, 5)};
  float nc = g.from(acc, 6);
  if (!act || g.sub != 0) return;
  if (!listed) {
    const RowWalk w(P, pi);
    walk_direct<true>(
        P, w, pi, i, pl, d.cellStart + P.cOff, d.bcellStart + P.cOff, d.bsample,
        [&](uint32_t, float4 q) {
          const F3 rij = sub3(pi, xyz(q));
          const float r2 = dot3(rij, rij);
          if (r2 < 1.0e-12f) return;
          dsum = fma3(fluid(r2, q.w), rij, dsum);
          nc += 1.0f;
        },
        [&](uint32_t, float4 q) {
          const F3 rij = sub3(pi, xyz(q));
          dB = fma3((self.w * q.w) * grad(dot3(rij, rij)), rij, dB);
        });
  }
  delta_finish(P, d, i, it, L, pi, dsum, dB, nc);
}

// xsph of one particle by a group (and, with N, the normals): sums x y z of xsph, then
// of the normal; terms: the xsph factor and velocity difference, the normal's factor and
// position difference.
template <int G, bool N, bool FAST>
__device__ __forceinline__ float group_xsph(const Group<G>& g, float (*sh)[N ? 9 : 5][kRow<G>], const SimParams& P,
                                            const DevScene& d, uint32_t i, bool act, const RowWalk& w, F3 pi, F3 vi,
                                            uint32_t* mine, const float4* __restrict__ pred, const uint32_t* __restrict__ cs,
                                            uint32_t& count) {
  count = act ? __ldg(&d.nbCount[i]) : kListOverflow;
  const bool keep = group_reusable(g, P, d, (int)P.iters, i, w, cell_index(P, w.c), count, act);  // every lane calls
  const bool need = act && !keep;
  count = group_build<G, false>(g, P, need, w, i, pi, pred, cs, nullptr, nullptr, mine, d.nbList, d.cap, P.h2,
                                count);
  const bool listed = act && count != kListOverflow;
  constexpr int NT = N ? 9 : 5;
  const int sa = g.sub < 3 ? 0 : 4, sb = g.sub < 3 ? 1 + g.sub : min(5 + (g.sub - 3), NT - 2);
  auto term = [&](float4 q, float4 v, float (&out)[NT]) {
    const F3 rij = sub3(pi, xyz(q));
    const float r2 = dot3(rij, rij);
    if (r2 >= P.h2) return;
    const float t = P.h2 - r2;
    const Root dens = density_of<FAST>(v.w);
    out[0] = over<FAST>(P.mass * (P.poly6 * t * t * t), dens);
    const F3 dv = sub3(xyz(v), vi);
    out[1] = dv.x;
    out[2] = dv.y;
    out[3] = dv.z;
    if constexpr (N) {
      if (r2 < 1.0e-12f) return;
      const Root rr = root_of<FAST>(r2);
      const float hr = P.h - rr.s;
      out[4] = over<FAST>(P.mass, dens) * over<FAST>(P.spikyGrad * hr * hr, rr);
      out[5] = rij.x;
      out[6] = rij.y;
      out[7] = rij.z;
    }
  };
  float acc = group_sums<G, NT, N ? 6 : 3, Pair4>(
      g, sh, d.nbList, d.cap, i, listed ? count & kCountMask : 0u, sa, sb, 0.0f,
      [&](uint32_t e) {
        const uint32_t j = (e & kBoundTag) != 0u ? i : e;  // walls have no part in these passes
        return Pair4{__ldg(&pred[j]), __ldg(&d.velRho[j])};
      },
      [&](uint32_t e, Pair4 p, float (&out)[NT]) {
        if ((e & kBoundTag) == 0u) term(p.q, p.g, out);
      });
  if (act && !listed) {  // every lane walks the reference's loop and keeps its own sum
    walk_direct<false>(
        P, w, pi, i, pred, cs, nullptr, nullptr,
        [&](uint32_t j, float4 q) {
          float out[NT];
#pragma unroll
          for (int s = 0; s < NT; s++) out[s] = 0.0f;
          term(q, __ldg(&d.velRho[j]), out);
          float a = 0.0f, b = 0.0f;
#pragma unroll
          for (int s = 0; s < NT; s++) {
            a = s == sa ? out[s] : a;
            b = s == sb ? out[s] : b;
          }
          acc = fmaf(a, b, acc);
        },
        [](uint32_t, float4) {});
  }
  __syncwarp();
  return acc;
}

template <int G, bool FAST>
__global__ void __launch_bounds__(kTB) k_xsph_finalize_g(const __grid_constant__ SimParams P,
                                                         const __grid_constant__ DevScene d) {
  __shared__ __align__(16) float sh[kTB / G][5][kRow<G>];
  __shared__ __align__(8) uint32_t lists[kTB / G][kListCap];
  const Group<G> g;
  const uint32_t li = (blockIdx.x * kTB + threadIdx.x) / G;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const float4 p4 = __ldg(&pred[i]);
  const F3 pi = xyz(p4), vi = xyz(__ldg(&d.vel[L ^ 1][i]));
  const RowWalk w(P, pi);
  uint32_t count;
  const float acc = group_xsph<G, false, FAST>(g, sh, P, d, i, act, w, pi, vi, lists[threadIdx.x / G], pred,
                                          d.cellStart + P.cOff, count);
  const F3 a = {g.from(acc, 0), g.from(acc, 1), g.from(acc, 2)};
  if (!act || g.sub != 0) return;
  const F3 vf = add3(vi, mul3(a, P.xsphC));
  d.vel[L][i] = make_float4(vf.x, vf.y, vf.z, 0.0f);
  d.pos[L][i] = p4;
  if ((P.iters & 1u) != 0u) d.pred[L][i] = p4;
}

template <int G, bool FAST>
__global__ void __launch_bounds__(kTB) k_xsph_normals_g(const __grid_constant__ SimParams P,
                                                        const __grid_constant__ DevScene d) {
  __shared__ __align__(16) float sh[kTB / G][9][kRow<G>];
  __shared__ __align__(8) uint32_t lists[kTB / G][kListCap];
  const Group<G> g;
  const uint32_t li = (blockIdx.x * kTB + threadIdx.x) / G;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const F3 pi = xyz(__ldg(&pred[i])), vi = xyz(__ldg(&d.vel[L ^ 1][i]));
  const RowWalk w(P, pi);
  uint32_t count;
  const float acc = group_xsph<G, true, FAST>(g, sh, P, d, i, act, w, pi, vi, lists[threadIdx.x / G], pred,
                                          d.cellStart + P.cOff, count);
  const F3 a = {g.from(acc, 0), g.from(acc, 1), g.from(acc, 2)}, n = {g.from(acc, 3), g.from(acc, 4), g.from(acc, 5)};
  if (!act || g.sub != 0) return;
  d.nbCount[i] = count;
  d.corr[i] = make_float4(P.xsphC * a.x, P.xsphC * a.y, P.xsphC * a.z, 0.0f);
  const F3 nrm = {P.h * n.x, P.h * n.y, P.h * n.z};
  d.normal[i] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
  d.normRho[i] = make_float4(nrm.x, nrm.y, nrm.z, __ldg(&d.density[i]));
}

template <int G, bool FAST>
__global__ void __launch_bounds__(kTB) k_tension_finalize_g(const __grid_constant__ SimParams P,
                                                            const __grid_constant__ DevScene d) {
  __shared__ __align__(16) float sh[kTB / G][5][kRow<G>];
  const Group<G> g;
  const uint32_t li = (blockIdx.x * kTB + threadIdx.x) / G;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const float4 p4 = __ldg(&pred[i]), n4 = __ldg(&d.normal[i]);
  const F3 pi = xyz(p4), ni = xyz(n4);
  const float rho = __ldg(&d.density[i]);
  const uint32_t count = act ? __ldg(&d.nbCount[i]) : 0u;
  const bool listed = act && count != kListOverflow;
  auto term = [&](float4 q, float4 v, float (&out)[5]) {
    const F3 rij = sub3(pi, xyz(q));
    const float r2 = dot3(rij, rij);
    if (r2 >= P.h2 || r2 < 1.0e-12f) return;
    const Root rt = root_of<FAST>(r2);
    const float rr = rt.s, hrr = P.h - rr;
    const float k = hrr * hrr * hrr * rr * rr * rr;
    float cw = P.cohes * (2.0f * k - P.cohesTerm);
    if (2.0f * rr > P.h) cw = P.cohes * k;
    const float sCoh = over<FAST>(-P.tension * P.mass * cw, rt);
    const F3 f = add3(mul3(rij, sCoh), mul3(sub3(ni, xyz(v)), -P.tension));
    out[0] = over<FAST>(2.0f * P.rho0, density_of<FAST>(rho + v.w));
    out[1] = f.x;
    out[2] = f.y;
    out[3] = f.z;
  };
  const int sb = min(1 + g.sub, 3);
  float acc = group_sums<G, 5, 3, Pair4>(
      g, sh, d.nbList, d.cap, i, listed ? count & kCountMask : 0u, 0, sb, 0.0f,
      [&](uint32_t e) {
        const uint32_t j = (e & kBoundTag) != 0u ? i : e;
        return Pair4{__ldg(&pred[j]), __ldg(&d.normRho[j])};
      },
      [&](uint32_t e, Pair4 p, float (&out)[5]) {
        if ((e & kBoundTag) == 0u) term(p.q, p.g, out);
      });
  if (act && !listed) {
    const RowWalk w(P, pi);
    walk_direct<false>(
        P, w, pi, i, pred, d.cellStart + P.cOff, nullptr, nullptr,
        [&](uint32_t j, float4 q) {
          float out[5] = {0.0f, 0.0f, 0.0f, 0.0f, 1.0f};
          term(q, __ldg(&d.normRho[j]), out);
          acc = fmaf(out[0], sb == 1 ? out[1] : sb == 2 ? out[2] : out[3], acc);
        },
        [](uint32_t, float4) {});
  }
  __syncwarp();
  const F3 a = {g.from(acc, 0), g.from(acc, 1), g.from(acc, 2)};
  if (!act || g.sub != 0) return;
  const float4 c0 = d.corr[i];
  const F3 cf = {fmaf(P.dt, a.x, c0.x), fmaf(P.dt, a.y, c0.y), fmaf(P.dt, a.z, c0.z)};
  d.corr[i] = make_float4(cf.x, cf.y, cf.z, 0.0f);
  const F3 vf = add3(xyz(__ldg(&d.vel[L ^ 1][i])), cf);
  d.vel[L][i] = make_float4(vf.x, vf.y, vf.z, 0.0f);
  d.pos[L][i] = p4;
  if ((P.iters & 1u) != 0u) d.pred[L][i] = p4;
}

template <int G>
static int group_blocks(const SimParams& P) { return groups((long long)P.n * G, kTB); }

#define P4A_GROUP_LAUNCH(K, flag, ...)                                                               \
  do {                                                                                               \
    const bool fast = (P.pairMath & (flag)) != 0u;                                                   \
    if (G == 16 && fast) K<16, true><<<group_blocks<16>(P), kTB, 0, st>>>(__VA_ARGS__);         \
    else if (fast) K<8, true><<<group_blocks<8>(P), kTB, 0, st>>>(__VA_ARGS__);                      \
    else K<8, false><<<group_blocks<8>(P), kTB, 0, st>>>(__VA_ARGS__);                               \
  } while (0)

void launch_lambda_g(const SimParams& P, const DevScene& d, int it, int G, cudaStream_t st) {
  P4A_GROUP_LAUNCH(k_lambda_g, PAIR_SOLVE, P, d, it);
}
void launch_delta_g(const SimParams& P, const DevScene& d, int it, int G, cudaStream_t st) {
  P4A_GROUP_LAUNCH(k_delta_g, PAIR_SOLVE, P, d, it);
}
void launch_xsph_finalize_g(const SimParams& P, const DevScene& d, int G, cudaStream_t st) {
  P4A_GROUP_LAUNCH(k_xsph_finalize_g, PAIR_XSPH, P, d);
}
void launch_xsph_normals_g(const SimParams& P, const DevScene& d, int G, cudaStream_t st) {
  P4A_GROUP_LAUNCH(k_xsph_normals_g, PAIR_XSPH, P, d);
}
void launch_tension_finalize_g(const SimParams& P, const DevScene& d, int G, cudaStream_t st) {
  P4A_GROUP_LAUNCH(k_tension_finalize_g, PAIR_TENSION, P, d);
}

}  // namespace p4a
