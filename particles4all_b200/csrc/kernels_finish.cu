// kernels_finish.cu — the 'finish' pass of a substep and the stats pass.
//   xsph       src/wgsl.js:85-123   (reads velFromPos velocities of neighbours)
//   normals    src/wgsl.js:250-288  (same neighbour walk as xsph: fused with it)
//   tension    src/wgsl.js:290-335
//   finalize   src/wgsl.js:337-350  (vel += corr; pos = pred), fused into the
//              last neighbour pass of the substep; the odd-k pred copy of
//              src/sim.js:568-573 is fused there too
//   stats      src/wgsl.js:785-832, fused into the last substep's finalize with
//              the reference's 256-particle workgroup trees, so the fixed-point
//              totals are the same bits
// With L = P.parity ^ 1 the live copy after the sort, the final positions are in
// pred[L ^ (iters & 1)]; the velFromPos velocities are in the non-live copy
// vel[L ^ 1], so the final velocity can be written to vel[L] while neighbours still
// read the other one. Each pass walks lambda's last list, or one it builds with radius
// h (neighbours.cuh); xsph+normals leaves the list for the tension pass, which walks
// the same positions. The pair terms run two at a time (pair_math.cuh); parameters
// outside its ranges take the IEEE operations on the same walk.
#include <cuda_runtime.h>

#include "neighbours.cuh"
#include "p4a_internal.h"
#include "p4a_math.cuh"
#include "pass_common.cuh"

namespace p4a {

// One 256-thread block's stats tree (src/wgsl.js:803-830): same pairings as the
// reference's shared-memory tree (shuffles reproduce them below 32).
__device__ __forceinline__ void block_stats(const SimParams& P, bool act, float dens, F3 v,
                                            uint32_t* __restrict__ out) {
  __shared__ float sR[kBlock], sM[kBlock], sV[kBlock], sK[kBlock];
  const int t = threadIdx.x;
  float rho = 0.0f, mrho = 0.0f, mv = 0.0f, ke = 0.0f;
  if (act) {
    rho = dens * P.invRho0;
    mrho = rho;
    const float v2 = dot3(v, v);
    mv = sqrtf(v2);
    ke = 0.5f * P.mass * v2;
  }
  sR[t] = rho; sM[t] = mrho; sV[t] = mv; sK[t] = ke;
  __syncthreads();
#pragma unroll
  for (int off = 128; off >= 32; off >>= 1) {
    if (t < off) {
      sR[t] = sR[t] + sR[t + off];
      sM[t] = fmaxf(sM[t], sM[t + off]);
      sV[t] = fmaxf(sV[t], sV[t + off]);
      sK[t] = sK[t] + sK[t + off];
    }
    __syncthreads();
  }
  if (t < 32) {
    float a = sR[t], b = sM[t], c = sV[t], e = sK[t];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a = a + __shfl_down_sync(0xffffffffu, a, off);
      b = fmaxf(b, __shfl_down_sync(0xffffffffu, b, off));
      c = fmaxf(c, __shfl_down_sync(0xffffffffu, c, off));
      e = e + __shfl_down_sync(0xffffffffu, e, off);
    }
    if (t == 0) {
      atomicAdd(&out[0], __float2uint_rz(a * 1024.0f));
      atomicMax(&out[1], __float2uint_rz(b * 1024.0f));
      atomicMax(&out[2], __float2uint_rz(c * 1024.0f));
      atomicAdd(&out[3], __float2uint_rz(e * 1024.0f));
    }
  }
}

// The neighbour list of the finishing passes (positions after the last Jacobi
// iteration): lambda's list when the displacement bound still covers it (its
// boundary samples are skipped by the walk: these passes have no boundary terms),
// else a new list with radius h, stored in nbList. `lanes` of the warp call: they come
// together again after the test, whose lanes return at four places, and after the builds;
// without that the builds ran once for each group (17 of 32 lanes active) and xsph of the
// preset took 60 us instead of 41, of 96 mixed scenes 238 instead of 216.
__device__ __forceinline__ uint32_t finish_list(const SimParams& P, const DevScene& d, const RowWalk& w,
                                                uint32_t i, F3 pi, const float4* __restrict__ pred,
                                                const uint32_t* __restrict__ cs, unsigned lanes) {
  uint32_t c = __ldg(&d.nbCount[i]);
  const bool reuse = list_reusable(P, d, (int)P.iters, i, w, cell_index(P, w.c), c);
  __syncwarp(lanes);
  if (!reuse) c = build_list<false>(P, w, i, pi, pred, cs, nullptr, nullptr, d.nbList, d.cap, P.h2);
  __syncwarp(lanes);
  return c;
}

// xsph (+ finalize) of scene-local particle li for scenes without surface
// tension; returns its density and final velocity for the stats (zero past the
// scene's end).
__device__ __forceinline__ void xsph_finalize_particle(const SimParams& P, const DevScene& d, uint32_t li,
                                                       float& rhoi, F3& vf) {
  vf = {0.f, 0.f, 0.f};
  rhoi = 0.0f;
  const unsigned lanes = __ballot_sync(0xffffffffu, li < P.n);
  if (li >= P.n) return;
  const uint32_t i = P.pOff + li;
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const float4* __restrict__ velIn = d.vel[L ^ 1];
  const uint32_t* __restrict__ cs = d.cellStart + P.cOff;
  const float4 p4 = __ldg(&pred[i]);
  const F3 pi = xyz(p4), vi = xyz(__ldg(&velIn[i]));
  const RowWalk w(P, pi);
  const uint32_t count = finish_list(P, d, w, i, pi, pred, cs, lanes);
  F3 acc = {0.f, 0.f, 0.f};
  // g = (velFromPos, max(density, rho0 / 2)) of neighbour j
  if (count != kListOverflow && (P.pairMath & PAIR_XSPH) != 0u) {
    const F2 h2 = splat2(P.h2), one = splat2(-1.0f), poly = splat2(P.poly6), mass = splat2(-P.mass);
    walk2g(d.nbList, d.cap, i, count, pred, d.velRho,
           [&](uint32_t j0, uint32_t j1, float4 q0, float4 q1, float4 g0, float4 g1) {
      const F3 r0 = sub3(pi, xyz(q0)), r1 = sub3(pi, xyz(q1));
      const float x0 = dot3(r0, r0), x1 = dot3(r1, r1);
      const bool in0 = !(x0 >= P.h2) && j0 != i, in1 = !(x1 >= P.h2) && j1 != i;
      const F2 dens = pack2(g0.w, g1.w);
      const F2 t = fma2(pack2(x0, x1), one, h2);
      const F2 f = quot2(mul2(mass, mul2(mul2(mul2(poly, t), t), t)), dens, recip2(dens));
      float f0, f1;
      unpack2(f, f0, f1);
      const F3 v0 = sub3(xyz(g0), vi), v1 = sub3(xyz(g1), vi);
      if (in0) acc = fma3(f0, v0, acc);
      if (in1) acc = fma3(f1, v1, acc);
    });
  } else {
    walk_fluid(P, w, i, pi, pred, d.velRho, cs, d.nbList, d.cap, count, [&](float4 q, float4 g) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2) return;  // in the skin of a reused list only
      const float t = P.h2 - r2;
      const float f = P.mass * (P.poly6 * t * t * t) / g.w;
      acc = fma3(f, sub3(xyz(g), vi), acc);
    });
  }
  const F3 corr = mul3(acc, P.xsphC);
  vf = add3(vi, corr);
  d.vel[L][i] = make_float4(vf.x, vf.y, vf.z, 0.0f);
  d.pos[L][i] = p4;
  if ((P.iters & 1u) != 0u) d.pred[L][i] = p4;
  rhoi = __ldg(&d.density[i]);
}

// Block form: 256-particle tile `tile`, with the stats tree after the last substep.
// All threads reach the tree, so there is no early return.
__device__ __forceinline__ void xsph_finalize_body(const SimParams& P, const DevScene& d, uint32_t tile,
                                                   int substep) {
  const uint32_t li = tile * kBlock + threadIdx.x;
  float rhoi;
  F3 vf;
  xsph_finalize_particle(P, d, li, rhoi, vf);
  if (substep == (int)P.subs - 1) block_stats(P, li < P.n, rhoi, vf, d.statsOut + 8 * P.slot);
}

// xsph + normals (tension scenes): corr = xsphC * acc, normal = h * nacc.
template <int TB>
__device__ __forceinline__ void xsph_normals_body(const SimParams& P, const DevScene& d, uint32_t li) {
  const unsigned lanes = __ballot_sync(0xffffffffu, li < P.n);
  if (li >= P.n) return;
  const uint32_t i = P.pOff + li;
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const float4* __restrict__ velIn = d.vel[L ^ 1];
  const uint32_t* __restrict__ cs = d.cellStart + P.cOff;
  const uint32_t cap = d.cap;
  const F3 pi = xyz(__ldg(&pred[i])), vi = xyz(__ldg(&velIn[i]));
  const RowWalk w(P, pi);
  const uint32_t count = finish_list(P, d, w, i, pi, pred, cs, lanes);
  d.nbCount[i] = count;
  F3 acc = {0.f, 0.f, 0.f}, nacc = {0.f, 0.f, 0.f};
  // g = (velFromPos, max(density, rho0 / 2)) of neighbour j
  if (count != kListOverflow && (P.pairMath & PAIR_XSPH) != 0u) {
    const F2 h2 = splat2(P.h2), h = splat2(P.h), one = splat2(-1.0f), poly = splat2(P.poly6);
    const F2 mass = splat2(-P.mass), cGrad = splat2(-P.spikyGrad);
    walk2g(d.nbList, cap, i, count, pred, d.velRho,
           [&](uint32_t j0, uint32_t j1, float4 q0, float4 q1, float4 g0, float4 g1) {
      const F3 r0 = sub3(pi, xyz(q0)), r1 = sub3(pi, xyz(q1));
      const float x0 = dot3(r0, r0), x1 = dot3(r1, r1);
      const bool in0 = !(x0 >= P.h2) && j0 != i, in1 = !(x1 >= P.h2) && j1 != i;
      const F2 x = pack2(x0, x1);
      const Root2 root = root2(x);
      const F2 dens = pack2(g0.w, g1.w), rd = recip2(dens);
      const F2 t = fma2(x, one, h2);
      const F2 f = quot2(mul2(mass, mul2(mul2(mul2(poly, t), t), t)), dens, rd);
      const F2 hr = fma2(root.s, one, h);
      const F2 grad = quot2(mul2(mul2(cGrad, hr), hr), root.s, root.yn);
      const F2 coef = mul2(quot2(mass, dens, rd), grad);
      float f0, f1, k0, k1;
      unpack2(f, f0, f1);
      unpack2(coef, k0, k1);
      const F3 v0 = sub3(xyz(g0), vi), v1 = sub3(xyz(g1), vi);
      if (in0) {
        acc = fma3(f0, v0, acc);
        if (!(x0 < 1.0e-12f)) nacc = fma3(k0, r0, nacc);
      }
      if (in1) {
        acc = fma3(f1, v1, acc);
        if (!(x1 < 1.0e-12f)) nacc = fma3(k1, r1, nacc);
      }
    });
  } else {
    walk_fluid(P, w, i, pi, pred, d.velRho, cs, d.nbList, cap, count, [&](float4 q, float4 g) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2) return;  // in the skin of a reused list only
      const float dj = g.w;
      const float t = P.h2 - r2;  // r2 < h2 here: poly6 without its range test
      const float f = P.mass * (P.poly6 * t * t * t) / dj;
      acc = fma3(f, sub3(xyz(g), vi), acc);
      if (r2 < 1.0e-12f) return;
      const float rr = sqrtf(r2);
      const float hr = P.h - rr;
      const float coef = (P.mass / dj) * (P.spikyGrad * hr * hr / rr);
      nacc = fma3(coef, rij, nacc);
    });
  }
  d.corr[i] = make_float4(P.xsphC * acc.x, P.xsphC * acc.y, P.xsphC * acc.z, 0.0f);
  const F3 nrm = {P.h * nacc.x, P.h * nacc.y, P.h * nacc.z};
  d.normal[i] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
  d.normRho[i] = make_float4(nrm.x, nrm.y, nrm.z, __ldg(&d.density[i]));  // for tension's gathers
}

// tension + finalize of scene-local particle li; density and final velocity out
// for the stats.
__device__ __forceinline__ void tension_finalize_particle(const SimParams& P, const DevScene& d, uint32_t li,
                                                          float& rhoi, F3& vf) {
  vf = {0.f, 0.f, 0.f};
  rhoi = 0.0f;
  const unsigned lanes = __ballot_sync(0xffffffffu, li < P.n);
  if (li >= P.n) return;
  const uint32_t i = P.pOff + li;
  const int L = (int)P.parity ^ 1;
  const float4* __restrict__ pred = d.pred[L ^ ((int)P.iters & 1)];
  const uint32_t* __restrict__ cs = d.cellStart + P.cOff;
  const uint32_t cap = d.cap;
  const float4 p4 = __ldg(&pred[i]);
  const F3 pi = xyz(p4), ni = xyz(__ldg(&d.normal[i]));
  const float rho = __ldg(&d.density[i]);
  const RowWalk w(P, pi);
  const uint32_t count = __ldg(&d.nbCount[i]);  // xsph+normals' list for these positions
  F3 acc = {0.f, 0.f, 0.f};
  // g = (normal, density) of neighbour j
  if (count != kListOverflow && (P.pairMath & PAIR_TENSION) != 0u) {
    const F2 h = splat2(P.h), one = splat2(-1.0f), two = splat2(2.0f), cohes = splat2(P.cohes);
    const F2 term = splat2(-P.cohesTerm), cCoh = splat2(P.tension * P.mass), cRho = splat2(-(2.0f * P.rho0));
    walk2g(d.nbList, cap, i, count, pred, d.normRho,
           [&](uint32_t, uint32_t, float4 q0, float4 q1, float4 g0, float4 g1) {
      const F3 r0 = sub3(pi, xyz(q0)), r1 = sub3(pi, xyz(q1));
      const float x0 = dot3(r0, r0), x1 = dot3(r1, r1);
      const bool in0 = !(x0 >= P.h2 || x0 < 1.0e-12f), in1 = !(x1 >= P.h2 || x1 < 1.0e-12f);
      const Root2 root = root2(pack2(x0, x1));
      const F2 hr = fma2(root.s, one, h);
      const F2 k = mul2(mul2(mul2(mul2(mul2(hr, hr), hr), root.s), root.s), root.s);
      float s0, s1, near0, near1, far0, far1;
      unpack2(root.s, s0, s1);
      unpack2(fma2(two, k, term), near0, near1);  // 2 k is exact
      unpack2(k, far0, far1);
      const F2 cw = mul2(cohes, pack2(2.0f * s0 > P.h ? far0 : near0, 2.0f * s1 > P.h ? far1 : near1));
      const F2 sCoh = quot2(mul2(cCoh, cw), root.s, root.yn);
      const F2 rhoSum = pack2(rho + g0.w, rho + g1.w);
      const F2 wgt = quot2(cRho, rhoSum, recip2(rhoSum));
      float c0, c1, w0, w1;
      unpack2(sCoh, c0, c1);
      unpack2(wgt, w0, w1);
      const F3 f0 = add3(mul3(r0, c0), mul3(sub3(ni, xyz(g0)), -P.tension));
      const F3 f1 = add3(mul3(r1, c1), mul3(sub3(ni, xyz(g1)), -P.tension));
      if (in0) acc = fma3(w0, f0, acc);
      if (in1) acc = fma3(w1, f1, acc);
    });
  } else {
    walk_fluid(P, w, i, pi, pred, d.normRho, cs, d.nbList, cap, count, [&](float4 q, float4 g) {
      const F3 rij = sub3(pi, xyz(q));
      const float r2 = dot3(rij, rij);
      if (r2 >= P.h2 || r2 < 1.0e-12f) return;
      const float rr = sqrtf(r2);
      const float hrr = P.h - rr;
      const float k = hrr * hrr * hrr * rr * rr * rr;
      float cw = P.cohes * (2.0f * k - P.cohesTerm);
      if (2.0f * rr > P.h) cw = P.cohes * k;
      const float sCoh = -P.tension * P.mass * cw / rr;
      const F3 fCoh = mul3(rij, sCoh);
      const F3 fCurv = mul3(sub3(ni, xyz(g)), -P.tension);
      const float wgt = 2.0f * P.rho0 / (rho + g.w);
      acc = fma3(wgt, add3(fCoh, fCurv), acc);
    });
  }
  const float4 c0 = d.corr[i];
  const F3 cf = {fmaf(P.dt, acc.x, c0.x), fmaf(P.dt, acc.y, c0.y), fmaf(P.dt, acc.z, c0.z)};
  d.corr[i] = make_float4(cf.x, cf.y, cf.z, 0.0f);
  const F3 vi = xyz(__ldg(&d.vel[L ^ 1][i]));
  vf = add3(vi, cf);
  d.vel[L][i] = make_float4(vf.x, vf.y, vf.z, 0.0f);
  d.pos[L][i] = p4;
  if ((P.iters & 1u) != 0u) d.pred[L][i] = p4;
  rhoi = rho;
}

__device__ __forceinline__ void tension_finalize_body(const SimParams& P, const DevScene& d,
                                                      uint32_t tile, int substep) {
  const uint32_t li = tile * kBlock + threadIdx.x;
  float rhoi;
  F3 vf;
  tension_finalize_particle(P, d, li, rhoi, vf);
  if (substep == (int)P.subs - 1) block_stats(P, li < P.n, rhoi, vf, d.statsOut + 8 * P.slot);
}

// Blocks of 256 per SM, which set the registers a thread may use. 5 (48 registers)
// spills the pair arithmetic: tension+finalize 469 us on the large scene against 267 us
// with 4 and 305 us with 3; batched on the 96-scene mix xsph+finalize 350 / 243 / 273 us
// and tension+finalize 574 / 302 / 284 us with 5 / 4 / 3.
constexpr int kFinishBlocks = 4, kTensionBlocksBatched = 3;
__global__ void __launch_bounds__(kBlock, kFinishBlocks) k_xsph_finalize(const __grid_constant__ SimParams P,
                                                             const __grid_constant__ DevScene d,
                                                             int substep) {
  xsph_finalize_body(P, d, blockIdx.x, substep);
}
__global__ void __launch_bounds__(kBlock, kFinishBlocks) k_xsph_finalize_b(const __grid_constant__ BatchWork w,
                                                               const __grid_constant__ DevScene d,
                                                               int substep) {
  for_each_item(w, [&](const SimParams& P, uint32_t t, uint32_t) { xsph_finalize_body(P, d, t, substep); });
}
template <int TB, int MB>
__global__ void __launch_bounds__(TB, MB) k_xsph_normals(const __grid_constant__ SimParams P,
                                                         const __grid_constant__ DevScene d, int) {
  xsph_normals_body<TB>(P, d, blockIdx.x * TB + threadIdx.x);
}
template <int TB, int MB>
__global__ void __launch_bounds__(TB, MB) k_xsph_normals_b(const __grid_constant__ BatchWork w,
                                                           const __grid_constant__ DevScene d, int) {
  for_each_slice(w, [&](const SimParams& P, uint32_t li) { xsph_normals_body<TB>(P, d, li); });
}
using PlainFn = void (*)(SimParams, DevScene, int);
using BatchFn = void (*)(BatchWork, DevScene, int);
static const PlainFn kNormalsP[kVariants] = {k_xsph_normals<256, 3>, k_xsph_normals<256, 4>,
                                             k_xsph_normals<256, 2>, k_xsph_normals<128, 6>,
                                             k_xsph_normals<128, 8>, k_xsph_normals<128, 5>};
static const BatchFn kNormalsB[kVariants] = {k_xsph_normals_b<256, 3>, k_xsph_normals_b<256, 4>,
                                             k_xsph_normals_b<256, 2>, k_xsph_normals_b<128, 6>,
                                             k_xsph_normals_b<128, 8>, k_xsph_normals_b<128, 5>};
__global__ void __launch_bounds__(kBlock, kFinishBlocks) k_tension_finalize(const __grid_constant__ SimParams P,
                                                                const __grid_constant__ DevScene d,
                                                                int substep) {
  tension_finalize_body(P, d, blockIdx.x, substep);
}
__global__ void __launch_bounds__(kBlock, kTensionBlocksBatched) k_tension_finalize_b(const __grid_constant__ BatchWork w,
                                                                  const __grid_constant__ DevScene d,
                                                                  int substep) {
  for_each_item(w, [&](const SimParams& P, uint32_t t, uint32_t) { tension_finalize_body(P, d, t, substep); });
}

// The stats pass on its own, for the group passes (kernels_group.cu), whose blocks are no
// tiles of 256 particles: the same trees over the stored densities and velocities.
__global__ void __launch_bounds__(kBlock) k_stats(const __grid_constant__ SimParams P,
                                                  const __grid_constant__ DevScene d) {
  const uint32_t li = blockIdx.x * kBlock + threadIdx.x;
  const bool act = li < P.n;
  const uint32_t i = P.pOff + (act ? li : 0u);
  block_stats(P, act, __ldg(&d.density[i]), xyz(__ldg(&d.vel[(int)P.parity ^ 1][i])), d.statsOut + 8 * P.slot);
}
void launch_stats(const SimParams& P, const DevScene& d, cudaStream_t st) {
  k_stats<<<groups(P.n), kBlock, 0, st>>>(P, d);
}

void launch_xsph_finalize(const SimParams& P, const DevScene& d, int substep, cudaStream_t st) {
  k_xsph_finalize<<<groups(P.n), kBlock, 0, st>>>(P, d, substep);
}
void launch_xsph_normals(const SimParams& P, const DevScene& d, cudaStream_t st, int variant) {
  const int v = variant >= 0 && variant < kVariants ? variant : tuned_variant(TK_NORMALS, P.n);
  const int tb = kShapes[TK_NORMALS][v].threads;
  kNormalsP[v]<<<groups(P.n, tb), tb, 0, st>>>(P, d, 0);
}
void launch_tension_finalize(const SimParams& P, const DevScene& d, int substep, cudaStream_t st) {
  k_tension_finalize<<<groups(P.n), kBlock, 0, st>>>(P, d, substep);
}
void launch_xsph_finalize_b(const BatchWork& w, int maxItems, const DevScene& d, int substep, cudaStream_t st) {
  k_xsph_finalize_b<<<persistent_grid((const void*)k_xsph_finalize_b, kBlock, maxItems), kBlock, 0, st>>>(w, d, substep);
}
void launch_xsph_normals_b(const BatchWork& w, int maxItems, const DevScene& d, cudaStream_t st, int variant) {
  const int v = variant >= 0 && variant < kVariants ? variant : tuned_variant(TK_NORMALS, (int64_t)maxItems * kBlock);
  const int tb = kShapes[TK_NORMALS][v].threads;
  kNormalsB[v]<<<persistent_grid((const void*)kNormalsB[v], tb, maxItems), tb, 0, st>>>(w, d, 0);
}
void launch_tension_finalize_b(const BatchWork& w, int maxItems, const DevScene& d, int substep,
                               cudaStream_t st) {
  k_tension_finalize_b<<<persistent_grid((const void*)k_tension_finalize_b, kBlock, maxItems), kBlock, 0, st>>>(w, d, substep);
}

}  // namespace p4a
