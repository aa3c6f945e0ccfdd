// kernels_solve.cu — the PBF Jacobi iteration: lambda (src/wgsl.js:477-543) and
// delta (src/wgsl.js:545-612). Gather-only: each thread owns one particle and visits
// the neighbours of the 3x3 row ranges around cellOf(current pred), using the
// cellStart of the substep's sort (the reference's stale-cell semantics), fluid then
// boundary samples per row, j ascending: the reference's accumulation order, so the
// sums are bit-identical to it under the float contract. No float atomics.
//
// Buffers follow the substep's parity L = P.parity ^ 1 (the live copy after the
// sort): iteration `it` reads pred[L ^ (it & 1)] and delta writes the other copy.
// lambda builds each particle's neighbour list (neighbours.cuh) with the radius
// h + skin and stores it; delta runs on the same positions and walks the same
// list. The list also serves later iterations of the substep: every delta (and
// the rigid projection) records the largest displacement of its iteration and the
// largest displacement from the substep's start positions, and a particle reuses
// its list while those bound every particle's movement since the list was built
// by skin / 2 (so every pair now within h was within h + skin then) and it is
// still in the cell it was in then (so its candidate rows are the same); see
// list_reusable. Every pass re-tests r^2 < h^2 on each listed candidate, so the
// visited neighbours and their order are exactly the reference's either way.
// The last delta of a substep also writes velFromPos (src/wgsl.js:72-83) for every
// particle into the non-live velocity copy; body particles are overwritten by the
// rigid projection that follows.
#include <cuda_runtime.h>

#include "neighbours.cuh"
#include "p4a_internal.h"
#include "p4a_math.cuh"
#include "pass_common.cuh"

namespace p4a {

// One list walk of lambda, two entries at a time; B: the list holds boundary samples
// (a fluid entry then takes the same path with its own coefficients selected, so that a
// warp at a wall runs every pair once and not once per kind). One entry at a time with the
// IEEE operations the walks were bound by issue slots (77 % of them busy, 80
// warp-instructions per entry, a quarter of those in the range tests of a root and a
// division): lambda took 728 us per launch on the 96-scene mix in halves, delta 426 us, on
// the large scene 289 and 232 us. With the packed pair arithmetic 525 and 327 us, 284 and
// 182 us; with the builds of neighbours.cuh and the prefetch of far_lists 492 and 297 us,
// 260 and 182 us. What bounds them now is the latency of the gathers (62 % of the slots, 49 %
// of the warps).
template <bool B, bool FAR>
__device__ __forceinline__ void lambda_walk(const SimParams& P, const DevScene& d, uint32_t i, uint32_t count, F3 pi,
                                            const float4* __restrict__ pred, float& rho, F3& gradSum,
                                            float& sumGrad2) {
  const F2 one = splat2(-1.0f), h2 = splat2(P.h2), h = splat2(P.h), poly = splat2(P.poly6);
  const F2 cFluid = splat2(-P.volSpiky);
  walk2<B, FAR>(d.nbList, d.cap, i, count, pred, d.bsample, [&](uint2 e, float4 q0, float4 q1) {
    const F3 r0 = sub3(pi, xyz(q0)), r1 = sub3(pi, xyz(q1));
    const float x0 = dot3(r0, r0), x1 = dot3(r1, r1);
    const bool b0 = B && (e.x & kBoundTag) != 0u, b1 = B && (e.y & kBoundTag) != 0u;
    const bool in0 = !(x0 >= P.h2 || (b0 && x0 < 1.0e-12f));
    const bool in1 = !(x1 >= P.h2 || (b1 && x1 < 1.0e-12f)) && e.y != i;
    const F2 x = pack2(x0, x1);
    const Root2 root = root2(x);
    const F2 t = fma2(x, one, h2);
    const F2 w = mul2(mul2(mul2(poly, t), t), t);
    const F2 hr = fma2(root.s, one, h);
    F2 c = cFluid;
    if constexpr (B)
      c = pack2(b0 ? -(q0.w * P.invRho0 * P.spikyGrad) : -P.volSpiky, b1 ? -(q1.w * P.invRho0 * P.spikyGrad) : -P.volSpiky);
    const F2 s = quot2(mul2(mul2(c, hr), hr), root.s, root.yn);
    float w0, w1, s0, s1;
    unpack2(w, w0, w1);
    unpack2(s, s0, s1);
    auto add = [&](bool in, bool b, float x, float psi, float wk, float sk, F3 r) {
      const F3 g = mul3(r, sk);
      const float g2 = dot3(g, g);
      if (in) {
        rho = fmaf(b ? psi : P.mass, wk, rho);
        if (b) {
          gradSum = fma3(sk, r, gradSum);
        } else if (x > 1.0e-12f) {
          gradSum = add3(gradSum, g);
          sumGrad2 = sumGrad2 + g2;
        }
      }
    };
    add(in0, b0, x0, q0.w, w0, s0, r0);
    add(in1, b1, x1, q1.w, w1, s1, r1);
  });
}

// Called by all 32 lanes of a warp (lanes past the scene's end only take part in the
// warp's list builds).
template <bool FAR>
__device__ __forceinline__ void lambda_body(const SimParams& P, const DevScene& d, uint32_t li, int it) {
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ (it & 1)];
  const uint32_t* __restrict__ cs = d.cellStart + P.cOff;
  const uint32_t* __restrict__ bcs = d.bcellStart + P.cOff;
  const uint32_t cap = d.cap;
  const F3 pi = xyz(__ldg(&pred[i]));
  const RowWalk w(P, pi);
  // reuse the stored list while the displacement bounds allow
  const uint32_t cell = cell_index(P, w.c);
  if (it == 0 && act) d.nbRef[i] = make_float4(pi.x, pi.y, pi.z, 0.0f);  // the substep's start positions
  uint32_t count = it > 0 && act ? __ldg(&d.nbCount[i]) : kListOverflow;
  const bool need = act && !list_reusable(P, d, it, i, w, cell, count);
  count = build_lists_warp<true>(P, need, w, i, pi, pred, cs, bcs, d.bsample, d.nbList, cap, P.skinH2, count);
  if (need) {
    if (count != kListOverflow) count |= (uint32_t)it << kBuildShift;
    d.nbCount[i] = count;
    d.nbCell[i] = cell;
  }
  if (!act) return;
  float rho = P.mass * poly6(P, 0.0f);
  F3 gradSum = {0.f, 0.f, 0.f};
  float sumGrad2 = 0.0f;
  if (count != kListOverflow && (P.pairMath & PAIR_SOLVE) != 0u) {
    // warps without a boundary sample in any list skip the kind selects
    if (__any_sync(__activemask(), (count & kHasBound) != 0u)) {
      lambda_walk<true, FAR>(P, d, i, count, pi, pred, rho, gradSum, sumGrad2);
    } else {
      lambda_walk<false, FAR>(P, d, i, count, pi, pred, rho, gradSum, sumGrad2);
    }
  } else {
    auto fluid = [&](uint32_t, float4 q) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2) return;  // in the skin of the list only
      const float t = P.h2 - r2;
      rho = fmaf(P.mass, P.poly6 * t * t * t, rho);  // poly6 within h
      if (r2 > 1.0e-12f) {
        const float rr = sqrtf(r2);
        const float hr = P.h - rr;
        const float s = P.volSpiky * hr * hr / rr;
        const F3 g = mul3(rij, s);
        gradSum = add3(gradSum, g);
        sumGrad2 = sumGrad2 + dot3(g, g);
      }
    };
    auto bound = [&](uint32_t, float4 q) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2 || r2 < 1.0e-12f) return;
      const float psi = q.w;
      const float t = P.h2 - r2;
      rho = fmaf(psi, P.poly6 * t * t * t, rho);
      const float rr = sqrtf(r2);
      const float hr = P.h - rr;
      const float s = psi * P.invRho0 * P.spikyGrad * hr * hr / rr;
      gradSum = fma3(s, rij, gradSum);
    };
    if (count != kListOverflow) {
      walk2<true, false>(d.nbList, cap, i, count, pred, d.bsample, [&](uint2 e, float4 q0, float4 q1) {
        if ((e.x & kBoundTag) != 0u) bound(e.x, q0);
        else fluid(e.x, q0);
        if ((e.y & kBoundTag) != 0u) bound(e.y, q1);
        else if (e.y != i) fluid(e.y, q1);
      });
    } else {
      walk_direct<true>(P, w, pi, i, pred, cs, bcs, d.bsample, fluid, bound);
    }
  }
  d.density[i] = rho;
  const float C = rho * P.invRho0 - 1.0f;
  float lam = 0.0f;
  if (C > 0.0f) {
    const float den = dot3(gradSum, gradSum) + sumGrad2 + P.cfmEps + 1.0e-12f;
    lam = -C / den;
  }
  d.lambda[i] = lam;
  // delta reads position and lambda of a neighbour with one 16-byte gather
  d.predLam[i] = make_float4(pi.x, pi.y, pi.z, lam);
}

// One list walk of delta, two entries at a time (B as in lambda_walk); nc counts the
// fluid neighbours for sorAverage.
template <bool B, bool FAR>
__device__ __forceinline__ void delta_walk(const SimParams& P, const DevScene& d, uint32_t i, uint32_t count,
                                           float4 self, F3& dsum, F3& dB, float& nc) {
  const F2 one = splat2(-1.0f), h2 = splat2(P.h2), h = splat2(P.h), poly = splat2(P.poly6);
  const F2 cGrad = splat2(-P.spikyGrad), wq = splat2(P.sCorrWq), kc = splat2(-P.sCorrK);
  const F3 pi = xyz(self);
  walk2<B, FAR>(d.nbList, d.cap, i, count, d.predLam, d.bsample, [&](uint2 e, float4 q0, float4 q1) {
    const F3 r0 = sub3(pi, xyz(q0)), r1 = sub3(pi, xyz(q1));
    const float x0 = dot3(r0, r0), x1 = dot3(r1, r1);
    const bool in0 = !(x0 >= P.h2 || x0 < 1.0e-12f), in1 = !(x1 >= P.h2 || x1 < 1.0e-12f);
    const F2 x = pack2(x0, x1);
    const Root2 root = root2(x);
    const F2 hr = fma2(root.s, one, h);
    const F2 s = quot2(mul2(mul2(cGrad, hr), hr), root.s, root.yn);
    const F2 t = fma2(x, one, h2);
    const F2 ratio = mul2(mul2(mul2(mul2(poly, t), t), t), wq);
    const F2 r2r = mul2(ratio, ratio);
    const F2 sc = mul2(mul2(kc, r2r), r2r);
    float c0, c1;
    unpack2(sc, c0, c1);
    const float f0 = self.w + q0.w + c0, f1 = self.w + q1.w + c1;
    if constexpr (B) {
      const bool b0 = (e.x & kBoundTag) != 0u, b1 = (e.y & kBoundTag) != 0u;
      float k0, k1;
      unpack2(mul2(pack2(b0 ? self.w * q0.w : f0, b1 ? self.w * q1.w : f1), s), k0, k1);
      auto add = [&](bool in, bool b, float coef, F3 r) {
        if (in && b) dB = fma3(coef, r, dB);
        if (in && !b) {
          dsum = fma3(coef, r, dsum);
          nc += 1.0f;
        }
      };
      add(in0, b0, k0, r0);
      add(in1, b1, k1, r1);
    } else {
      float k0, k1;
      unpack2(mul2(pack2(f0, f1), s), k0, k1);
      if (in0) {
        dsum = fma3(k0, r0, dsum);
        nc += 1.0f;
      }
      if (in1) {
        dsum = fma3(k1, r1, dsum);
        nc += 1.0f;
      }
    }
  });
}

template <bool FAR>
__device__ __forceinline__ void delta_body(const SimParams& P, const DevScene& d, uint32_t li, int it) {
  if (li >= P.n) return;
  const uint32_t i = P.pOff + li;
  const int L = (int)P.parity ^ 1;
  // lambda's (position, lambda) of this iteration: the positions of pred[L ^ (it & 1)]
  const float4* __restrict__ pl = d.predLam;
  const float4 self = __ldg(&pl[i]);
  const F3 pi = xyz(self);
  const uint32_t count = __ldg(&d.nbCount[i]);  // lambda's list for these positions
  F3 dsum = {0.f, 0.f, 0.f}, dB = {0.f, 0.f, 0.f};
  float nc = 1.0f;
  if (count != kListOverflow && (P.pairMath & PAIR_SOLVE) != 0u) {
    if (__any_sync(__activemask(), (count & kHasBound) != 0u)) {
      delta_walk<true, FAR>(P, d, i, count, self, dsum, dB, nc);
    } else {
      delta_walk<false, FAR>(P, d, i, count, self, dsum, dB, nc);
    }
  } else {
    const float li_ = self.w;
    auto fluid = [&](uint32_t, float4 q) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2 || r2 < 1.0e-12f) return;
      const float rr = sqrtf(r2);
      const float hr = P.h - rr;
      const float s = P.spikyGrad * hr * hr / rr;
      const float t = P.h2 - r2;
      const float ratio = P.poly6 * t * t * t * P.sCorrWq;
      const float r2r = ratio * ratio;
      const float sc = -P.sCorrK * r2r * r2r;
      const float coef = (li_ + q.w + sc) * s;
      dsum = fma3(coef, rij, dsum);
      nc += 1.0f;
    };
    auto bound = [&](uint32_t, float4 q) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2 || r2 < 1.0e-12f) return;
      const float rr = sqrtf(r2);
      const float hr = P.h - rr;
      const float coef = (li_ * q.w) * (P.spikyGrad * hr * hr / rr);
      dB = fma3(coef, rij, dB);
    };
    if (count != kListOverflow) {
      walk2<true, false>(d.nbList, d.cap, i, count, pl, d.bsample, [&](uint2 e, float4 q0, float4 q1) {
        if ((e.x & kBoundTag) != 0u) bound(e.x, q0);
        else fluid(e.x, q0);
        if ((e.y & kBoundTag) != 0u) bound(e.y, q1);
        else if (e.y != i) fluid(e.y, q1);
      });
    } else {
      const RowWalk w(P, pi);
      walk_direct<true>(P, w, pi, i, pl, d.cellStart + P.cOff, d.bcellStart + P.cOff, d.bsample, fluid, bound);
    }
  }
  delta_finish(P, d, i, it, L, pi, dsum, dB, nc);
}

// Plain: block b handles particles [b * TB, (b + 1) * TB). Batched: warps pull
// 32-particle slices of the segment's tiles.
template <int TB, int MB, bool FAR>
__global__ void __launch_bounds__(TB, MB) k_lambda(const __grid_constant__ SimParams P,
                                                   const __grid_constant__ DevScene d, int it) {
  lambda_body<FAR>(P, d, blockIdx.x * TB + threadIdx.x, it);
}
template <int TB, int MB>
__global__ void __launch_bounds__(TB, MB) k_lambda_b(const __grid_constant__ BatchWork w,
                                                     const __grid_constant__ DevScene d, int it) {
  for_each_slice(w, [&](const SimParams& P, uint32_t li) { lambda_body<false>(P, d, li, it); });
}
template <int TB, int MB>
__global__ void __launch_bounds__(TB, MB) k_delta(const __grid_constant__ SimParams P,
                                                  const __grid_constant__ DevScene d, int it) {
  delta_body<false>(P, d, blockIdx.x * TB + threadIdx.x, it);
}
template <int TB, int MB, bool FAR>
__global__ void __launch_bounds__(TB, MB) k_delta_b(const __grid_constant__ BatchWork w,
                                                    const __grid_constant__ DevScene d, int it) {
  for_each_slice(w, [&](const SimParams& P, uint32_t li) { delta_body<FAR>(P, d, li, it); });
}

using PlainFn = void (*)(SimParams, DevScene, int);
using BatchFn = void (*)(BatchWork, DevScene, int);
#define P4A_SHAPES(K, ...)                                                                           \
  {K<256, 4 __VA_ARGS__>, K<256, 3 __VA_ARGS__>, K<256, 5 __VA_ARGS__>, K<128, 8 __VA_ARGS__>,       \
   K<128, 6 __VA_ARGS__>, K<128, 10 __VA_ARGS__>}
#define P4A_FAR(x) , x
static const PlainFn kLambdaP[2][kVariants] = {P4A_SHAPES(k_lambda, P4A_FAR(false)),
                                               P4A_SHAPES(k_lambda, P4A_FAR(true))};
static const BatchFn kLambdaB[kVariants] = P4A_SHAPES(k_lambda_b);
static const PlainFn kDeltaP[kVariants] = P4A_SHAPES(k_delta);
static const BatchFn kDeltaB[2][kVariants] = {P4A_SHAPES(k_delta_b, P4A_FAR(false)),
                                              P4A_SHAPES(k_delta_b, P4A_FAR(true))};

static int pick(int kernel, int variant, int64_t n) {
  return variant >= 0 && variant < kVariants ? variant : tuned_variant(kernel, n);
}

void launch_lambda(const SimParams& P, const DevScene& d, int it, cudaStream_t st, int variant) {
  const int v = pick(TK_LAMBDA, variant, P.n), tb = kShapes[TK_LAMBDA][v].threads;
  kLambdaP[far_lists(P.n)][v]<<<groups(P.n, tb), tb, 0, st>>>(P, d, it);
}
void launch_delta(const SimParams& P, const DevScene& d, int it, cudaStream_t st, int variant) {
  const int v = pick(TK_DELTA, variant, P.n), tb = kShapes[TK_DELTA][v].threads;
  kDeltaP[v]<<<groups(P.n, tb), tb, 0, st>>>(P, d, it);
}
void launch_lambda_b(const BatchWork& w, int maxItems, const DevScene& d, int it, cudaStream_t st, int variant) {
  const int v = pick(TK_LAMBDA, variant, (int64_t)maxItems * kBlock), tb = kShapes[TK_LAMBDA][v].threads;
  kLambdaB[v]<<<persistent_grid((const void*)kLambdaB[v], tb, maxItems), tb, 0, st>>>(w, d, it);
}
void launch_delta_b(const BatchWork& w, int maxItems, const DevScene& d, int it, bool far, cudaStream_t st,
                    int variant) {
  const int v = pick(TK_DELTA, variant, (int64_t)maxItems * kBlock), tb = kShapes[TK_DELTA][v].threads;
  const BatchFn k = kDeltaB[far][v];
  k<<<persistent_grid((const void*)k, tb, maxItems), tb, 0, st>>>(w, d, it);
}

}  // namespace p4a
