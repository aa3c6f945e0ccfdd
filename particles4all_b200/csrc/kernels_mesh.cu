// kernels_mesh.cu — the surface mesh of the simulation (src/mesh_wgsl.js:23-238,
// driven by src/mesh.js:99-340): a density field on the vertices of a voxel grid
// gathered from the particles, 3-tap blur passes, and marching tetrahedra (six
// tetrahedra per voxel) emitting triangles as packed vertices (16-bit grid
// position, octahedral normal).
//
// The reference appends triangles through an atomic counter, so its triangle order
// is whatever the atomics produce. Here a count pass, the decoupled-lookback scan of
// kernels_grid.cu (over the triangle counts of blocks of 256 voxels) and an emit pass
// write them in voxel order (tetrahedra and quad halves in the reference's order
// within a voxel): the same triangles, in one fixed order, and the total is the count
// the reference's counter reaches.
#include <cuda_runtime.h>

#include "p4a_internal.h"
#include "p4a_math.cuh"

namespace p4a {

__device__ __forceinline__ I3 grid_vertex(const MeshParams& M, uint32_t idx, const int32_t dim[3]) {
  I3 v;
  v.x = (int)(idx % (uint32_t)dim[0]);
  v.y = (int)((idx / (uint32_t)dim[0]) % (uint32_t)dim[1]);
  v.z = (int)(idx / ((uint32_t)dim[0] * (uint32_t)dim[1]));
  return v;
}

// What meshDensity reads of particle j for every vertex around it: its position and
// (mass / max(rho, rho0 / 2)) * poly6. A body particle that is skipped counts as infinitely
// far away, so that it adds nothing whatever its position (NaN among them). Formed once
// per particle: in the gather below each was recomputed, with its division, for some 500
// candidate tests per particle (221 us per field of the 250,000-particle scene on
// 131 x 131 x 89 vertices).
__global__ void __launch_bounds__(kBlock) k_mesh_weights(const __grid_constant__ MeshParams M,
                                                         const float4* __restrict__ pos,
                                                         const float* __restrict__ rho,
                                                         const uint4* __restrict__ body, uint32_t n,
                                                         float4* __restrict__ out) {
  const uint32_t j = blockIdx.x * kBlock + threadIdx.x;
  if (j >= n) return;
  const float4 p = __ldg(&pos[j]);
  const bool skip = M.skipBodies != 0u && __ldg(&body[j]).x != 0u;
  const float vol = M.mass / fmaxf(__ldg(&rho[j]), 0.5f * M.rho0);
  out[j] = skip ? make_float4(INFINITY, INFINITY, INFINITY, 0.0f) : make_float4(p.x, p.y, p.z, vol * M.poly6);
}

// meshDensity (src/mesh_wgsl.js:23-69). A block takes 8 x 8 x 4 vertices and a warp
// 4 x 4 x 2 of them, a cube of a few cells, so that its lanes walk nearly the same
// candidates (a warp of 32 vertices along x spans some 15 cells, whose gathers share
// nothing: 125 us against 97 us on 131 x 131 x 89 vertices).
__global__ void __launch_bounds__(kBlock) k_mesh_field(const __grid_constant__ MeshParams M,
                                                       const float4* __restrict__ weights,
                                                       const uint32_t* __restrict__ cs, uint32_t n,
                                                       float* __restrict__ field) {
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
  const I3 v = {(int)blockIdx.x * 8 + (warp & 1) * 4 + (lane & 3), (int)blockIdx.y * 8 + (warp >> 1 & 1) * 4 + (lane >> 2 & 3),
                (int)blockIdx.z * 4 + (warp >> 2) * 2 + (lane >> 4)};
  if (v.x >= M.vertDim[0] || v.y >= M.vertDim[1] || v.z >= M.vertDim[2]) return;
  const F3 p = {M.gridOrigin[0] + M.voxel * (float)v.x, M.gridOrigin[1] + M.voxel * (float)v.y,
                M.gridOrigin[2] + M.voxel * (float)v.z};
  I3 c;
  c.x = min(max(__float2int_rz(floorf((p.x - M.boxMin[0]) * M.invSupport)), 0), M.simGridDim[0] - 1);
  c.y = min(max(__float2int_rz(floorf((p.y - M.boxMin[1]) * M.invSupport)), 0), M.simGridDim[1] - 1);
  c.z = min(max(__float2int_rz(floorf((p.z - M.boxMin[2]) * M.invSupport)), 0), M.simGridDim[2] - 1);
  const int x0 = max(c.x - 1, 0), x1 = min(c.x + 1, M.simGridDim[0] - 1);
  // the nine rows' bounds first, every load independent of the others
  uint32_t rb[9], re[9];
#pragma unroll
  for (int r = 0; r < 9; r++) {
    const int z = c.z + r / 3 - 1, y = c.y + r % 3 - 1;
    const bool in = z >= 0 && z < M.simGridDim[2] && y >= 0 && y < M.simGridDim[1];
    const uint32_t rowBase = in ? (uint32_t)((z * M.simGridDim[1] + y) * M.simGridDim[0]) : 0u;
    rb[r] = __ldg(&cs[rowBase + x0]);
    re[r] = in ? min(__ldg(&cs[rowBase + x1 + 1]), n) : 0u;
  }
  float acc = 0.0f;
  auto add = [&](float4 q) {
    const F3 r = sub3(p, xyz(q));
    const float r2 = dot3(r, r);
    const float t = M.support2 - r2;
    if (!(r2 >= M.support2)) acc = fmaf((q.w * t) * t, t, acc);
  };
#pragma unroll
  for (int r = 0; r < 9; r++) {
    uint32_t j = rb[r];
    for (; j + 4 <= re[r]; j += 4) {
      const float4 q0 = __ldg(&weights[j]), q1 = __ldg(&weights[j + 1]);
      const float4 q2 = __ldg(&weights[j + 2]), q3 = __ldg(&weights[j + 3]);
      add(q0);
      add(q1);
      add(q2);
      add(q3);
    }
    for (; j < re[r]; j++) add(__ldg(&weights[j]));
  }
  field[((uint32_t)v.z * M.vertDim[1] + v.y) * M.vertDim[0] + v.x] = acc;
}

// meshSmooth (src/mesh_wgsl.js:71-92) along one axis, `passes` times in a row: one
// warp per grid line, the line held in shared memory (two buffers of `len` floats
// per warp), clamped at the ends like the reference's S().
__global__ void __launch_bounds__(128) k_mesh_blur(const float* __restrict__ src, float* __restrict__ dst,
                                                   int dx, int dy, int dz, int axis, int passes, int lines) {
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int line = blockIdx.x * 4 + warp;
  if (line >= lines) return;  // whole warps
  const int len = axis == 0 ? dx : axis == 1 ? dy : dz;
  float* a = smem + (size_t)warp * 2 * len;
  float* b = a + len;
  size_t base, stride;
  if (axis == 0) {
    base = (size_t)line * dx;
    stride = 1;
  } else if (axis == 1) {
    base = (size_t)(line / dx) * dx * dy + (size_t)(line % dx);
    stride = (size_t)dx;
  } else {
    base = (size_t)line;
    stride = (size_t)dx * dy;
  }
  for (int k = lane; k < len; k += 32) a[k] = src[base + k * stride];
  __syncwarp();
  for (int p = 0; p < passes; p++) {
    for (int k = lane; k < len; k += 32) {
      const float l = a[max(k - 1, 0)], m = a[k], r = a[min(k + 1, len - 1)];
      b[k] = (0.25f * l + 0.5f * m) + 0.25f * r;
    }
    __syncwarp();
    float* t = a;
    a = b;
    b = t;
  }
  for (int k = lane; k < len; k += 32) dst[base + k * stride] = a[k];
}

// ---- marching tetrahedra (src/mesh_wgsl.js:94-238) ---------------------------

__device__ __forceinline__ float field_at(const float* __restrict__ f, const MeshParams& M, I3 v) {
  v.x = min(max(v.x, 0), M.vertDim[0] - 1);
  v.y = min(max(v.y, 0), M.vertDim[1] - 1);
  v.z = min(max(v.z, 0), M.vertDim[2] - 1);
  return __ldg(&f[(uint32_t)((v.z * M.vertDim[1] + v.y) * M.vertDim[0] + v.x)]);
}

__device__ __forceinline__ F3 grad_at(const float* __restrict__ nf, const MeshParams& M, I3 v) {
  return {field_at(nf, M, {v.x + 1, v.y, v.z}) - field_at(nf, M, {v.x - 1, v.y, v.z}),
          field_at(nf, M, {v.x, v.y + 1, v.z}) - field_at(nf, M, {v.x, v.y - 1, v.z}),
          field_at(nf, M, {v.x, v.y, v.z + 1}) - field_at(nf, M, {v.x, v.y, v.z - 1})};
}

struct Corner {
  float d;
  F3 p, g;
};

__device__ __forceinline__ uint32_t to_u32(float x) { return __float2uint_rz(x); }

__device__ __forceinline__ uint2 pack_vertex(const MeshParams& M, F3 pg, F3 nIn) {
  const F3 pn = {fminf(fmaxf(pg.x / (float)(M.vertDim[0] - 1), 0.0f), 1.0f),
                 fminf(fmaxf(pg.y / (float)(M.vertDim[1] - 1), 0.0f), 1.0f),
                 fminf(fmaxf(pg.z / (float)(M.vertDim[2] - 1), 0.0f), 1.0f)};
  const uint32_t qx = to_u32(pn.x * 65535.0f + 0.5f), qy = to_u32(pn.y * 65535.0f + 0.5f),
                 qz = to_u32(pn.z * 65535.0f + 0.5f);
  const float l1 = fmaxf((fabsf(nIn.x) + fabsf(nIn.y)) + fabsf(nIn.z), 1.0e-12f);
  const F3 nv = {nIn.x / l1, nIn.y / l1, nIn.z / l1};
  float ex = nv.x, ey = nv.y;
  if (nv.z < 0.0f) {
    ex = (1.0f - fabsf(nv.y)) * (nv.x >= 0.0f ? 1.0f : -1.0f);
    ey = (1.0f - fabsf(nv.x)) * (nv.y >= 0.0f ? 1.0f : -1.0f);
  }
  const uint32_t ox = to_u32(fminf(fmaxf(ex * 0.5f + 0.5f, 0.0f), 1.0f) * 255.0f + 0.5f);
  const uint32_t oy = to_u32(fminf(fmaxf(ey * 0.5f + 0.5f, 0.0f), 1.0f) * 255.0f + 0.5f);
  return make_uint2(qx | (qy << 16), qz | ((ox | (oy << 8)) << 16));
}

// mix(x, y, t) = x * (1 - t) + y * t
__device__ __forceinline__ F3 mix3(F3 x, F3 y, float t) {
  const float s = 1.0f - t;
  return {x.x * s + y.x * t, x.y * s + y.y * t, x.z * s + y.z * t};
}

__device__ __forceinline__ uint2 edge_vertex(const MeshParams& M, const Corner& a, const Corner& b) {
  const float t = (M.iso - a.d) / (b.d - a.d);
  const F3 p = mix3(a.p, b.p, t);
  const F3 g = mix3(a.g, b.g, t);
  return pack_vertex(M, p, {-g.x, -g.y, -g.z});
}

// Triangles of one tetrahedron (emitTet): 0, 1 (one corner in or out) or 2 (a quad).
__device__ __forceinline__ int tet_triangles(bool ia, bool ib, bool ic, bool id) {
  const int nin = (int)ia + (int)ib + (int)ic + (int)id;
  return nin == 0 || nin == 4 ? 0 : nin == 2 ? 2 : 1;
}

// The six tetrahedra of a voxel, corners (0,1,3,7) (0,1,5,7) (0,2,3,7) (0,2,6,7)
// (0,4,5,7) (0,4,6,7); corner k = (k & 1, k >> 1 & 1, k >> 2 & 1). The middle corners of
// tetrahedron t are nibble t of these words.
constexpr uint32_t kTetB = 0x442211u, kTetC = 0x656353u;
__device__ __forceinline__ int tet_corner(int t, int k) {
  return k == 0 ? 0 : k == 3 ? 7 : (int)(((k == 1 ? kTetB : kTetC) >> (4 * t)) & 7u);
}
// Triangles of tetrahedron t of a voxel with corner signs `mask`.
__device__ __forceinline__ uint32_t tet_count(uint32_t mask, int t) {
  return (uint32_t)tet_triangles((mask & 1u) != 0u, ((mask >> tet_corner(t, 1)) & 1u) != 0u,
                                 ((mask >> tet_corner(t, 2)) & 1u) != 0u, ((mask >> 7) & 1u) != 0u);
}

__device__ __forceinline__ I3 voxel_of(const MeshParams& M, uint32_t idx) {
  const int32_t nv[3] = {M.vertDim[0] - 1, M.vertDim[1] - 1, M.vertDim[2] - 1};
  return grid_vertex(M, idx, nv);
}

// Per voxel: the corner signs and the triangle count. A voxel with triangles is appended
// to `active` as (voxel, signs | triangles of the block's earlier voxels << 8), in any
// order; the block's total goes to blockSum for the scan. Emitting from the list keeps
// its warps full: 6 % of the voxels have triangles, and a thread per voxel left most
// lanes of every warp idle (222 us for 271,000 triangles).
__global__ void __launch_bounds__(kBlock) k_mesh_count(const __grid_constant__ MeshParams M,
                                                       const float* __restrict__ field,
                                                       uint32_t* __restrict__ blockSum, uint2* __restrict__ active,
                                                       uint32_t* __restrict__ activeCount, uint32_t nvox) {
  __shared__ uint32_t sWarp[kBlock / 32];
  const uint32_t idx = blockIdx.x * kBlock + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t mask = 0u, c = 0u;
  if (idx < nvox) {
    const I3 v = voxel_of(M, idx);
#pragma unroll
    for (int k = 0; k < 8; k++)
      mask |= (field_at(field, M, {v.x + (k & 1), v.y + ((k >> 1) & 1), v.z + ((k >> 2) & 1)}) > M.iso ? 1u : 0u) << k;
    if (mask != 0u && mask != 255u) {
#pragma unroll
      for (int t = 0; t < 6; t++) c += tet_count(mask, t);
    }
  }
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += t;
  }
  if (lane == 31u) sWarp[warp] = incl;
  __syncthreads();
  uint32_t before = 0u, total = 0u;
#pragma unroll
  for (uint32_t w = 0; w < kBlock / 32; w++) {
    before += w < warp ? sWarp[w] : 0u;
    total += sWarp[w];
  }
  if (threadIdx.x == 0) blockSum[blockIdx.x] = total;
  const uint32_t m = __ballot_sync(0xffffffffu, c != 0u);
  if (m == 0u) return;
  uint32_t base = 0u;
  if (lane == 0u) base = atomicAdd(activeCount, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (c != 0u)
    active[base + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(idx, mask | ((before + incl - c) << 8));
}

// Marching tetrahedra of the listed voxels: a warp takes one tetrahedron of 32 of them.
// A lone corner l (in or out) against p1, p2, p3 gives the triangle of the edges (l, p1),
// (l, p2), (l, p3); two corners a, b in and c, d out give the quad of the edges (a, c),
// (a, d), (b, d), (b, c) as triangles 0 1 2 and 0 2 3; corners in ascending order.
__global__ void __launch_bounds__(128) k_mesh_emit(const __grid_constant__ MeshParams M,
                                                   const float* __restrict__ field,
                                                   const float* __restrict__ nfield,
                                                   const uint32_t* __restrict__ blockOffset,
                                                   const uint2* __restrict__ active,
                                                   const uint32_t* __restrict__ activeCount,
                                                   uint2* __restrict__ verts) {
  __shared__ float sc[4][7][128];  // [corner][d, p, g][thread]
  const uint32_t count = *activeCount, lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * 4u, tasks = (count + 31u) / 32u * 6u;
  for (uint32_t task = blockIdx.x * 4u + (threadIdx.x >> 5); task < tasks; task += warps) {
    const int t = (int)(task % 6u);
    const uint32_t a = task / 6u * 32u + lane;
    if (a >= count) continue;
    const uint2 en = __ldg(&active[a]);
    const uint32_t mask = en.y & 255u, tris = tet_count(mask, t);
    if (tris == 0u) continue;
    uint32_t at = blockOffset[en.x / kBlock] + (en.y >> 8);
    for (int k = 0; k < t; k++) at += tet_count(mask, k);
    if (at >= M.maxTris) continue;
    const I3 v = voxel_of(M, en.x);
    uint32_t in = 0u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int cr = tet_corner(t, k);
      const I3 w = {v.x + (cr & 1), v.y + ((cr >> 1) & 1), v.z + ((cr >> 2) & 1)};
      const F3 g = grad_at(nfield, M, w);
      in |= ((mask >> cr) & 1u) << k;
      sc[k][0][threadIdx.x] = field_at(field, M, w);
      sc[k][1][threadIdx.x] = (float)w.x;
      sc[k][2][threadIdx.x] = (float)w.y;
      sc[k][3][threadIdx.x] = (float)w.z;
      sc[k][4][threadIdx.x] = g.x;
      sc[k][5][threadIdx.x] = g.y;
      sc[k][6][threadIdx.x] = g.z;
    }
    // the edges as two nibbles each, first edge lowest
    uint32_t edges;
    if (tris == 1u) {
      const uint32_t lone = __popc(in) == 1 ? in : in ^ 15u, l = (uint32_t)__ffs(lone) - 1u, rest = lone ^ 15u;
      const uint32_t p1 = (uint32_t)__ffs(rest) - 1u, p2 = (uint32_t)__ffs(rest & (rest - 1u)) - 1u, p3 = 6u - l - p1 - p2;
      edges = l * 0x010101u | p1 << 4 | p2 << 12 | p3 << 20;
    } else {
      const uint32_t out = in ^ 15u;
      const uint32_t qa = (uint32_t)__ffs(in) - 1u, qb = 31u - (uint32_t)__clz(in);
      const uint32_t qc = (uint32_t)__ffs(out) - 1u, qd = 31u - (uint32_t)__clz(out);
      edges = qa | qc << 4 | qa << 8 | qd << 12 | qb << 16 | qd << 20 | qb << 24 | qc << 28;
    }
    const bool second = tris == 2u && at + 1u < M.maxTris;
    uint2* __restrict__ o = verts + (size_t)at * 3;
#pragma unroll 1
    for (uint32_t k = 0; k < (second ? 4u : 3u); k++) {
      const uint32_t ka = (edges >> (8u * k)) & 15u, kb = (edges >> (8u * k + 4u)) & 15u;
      auto corner = [&](uint32_t q) {
        return Corner{sc[q][0][threadIdx.x],
                      {sc[q][1][threadIdx.x], sc[q][2][threadIdx.x], sc[q][3][threadIdx.x]},
                      {sc[q][4][threadIdx.x], sc[q][5][threadIdx.x], sc[q][6][threadIdx.x]}};
      };
      const uint2 vert = edge_vertex(M, corner(ka), corner(kb));
      if (k < 3u) o[k] = vert;
      if (second && k == 0u) o[3] = vert;
      if (second && k >= 2u) o[k + 2u] = vert;
    }
  }
}

void launch_mesh_field(const MeshParams& M, const float4* pos, const float* rho, const uint32_t* cs,
                       const uint4* body, uint32_t n, float4* weights, float* field, cudaStream_t st) {
  const dim3 grid((M.vertDim[0] + 7) / 8, (M.vertDim[1] + 7) / 8, (M.vertDim[2] + 3) / 4);
  count_launches(1);
  k_mesh_weights<<<groups(n), kBlock, 0, st>>>(M, pos, rho, body, n, weights);
  k_mesh_field<<<grid, kBlock, 0, st>>>(M, weights, cs, n, field);
}

cudaError_t launch_mesh_blur(const MeshParams& M, const float* src, float* dst, int axis, int passes,
                             cudaStream_t st) {
  const int dx = M.vertDim[0], dy = M.vertDim[1], dz = M.vertDim[2];
  const int len = axis == 0 ? dx : axis == 1 ? dy : dz;
  const int lines = (dx * dy * dz) / len;
  const size_t smem = (size_t)4 * 2 * len * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k_mesh_blur, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_mesh_blur<<<(lines + 3) / 4, 128, smem, st>>>(src, dst, dx, dy, dz, axis, passes, lines);
  return cudaGetLastError();
}

void launch_mesh_count(const MeshParams& M, const float* field, uint32_t* blockSum, uint2* active,
                       uint32_t* activeCount, uint32_t nvox, cudaStream_t st) {
  cudaMemsetAsync(activeCount, 0, 4, st);
  k_mesh_count<<<groups(nvox), kBlock, 0, st>>>(M, field, blockSum, active, activeCount, nvox);
}

void launch_mesh_emit(const MeshParams& M, const float* field, const float* nfield, const uint32_t* blockOffset,
                      const uint2* active, const uint32_t* activeCount, uint2* verts, cudaStream_t st) {
  count_launches(1);
  k_mesh_emit<<<148 * 12, 128, 0, st>>>(M, field, nfield, blockOffset, active, activeCount, verts);
}

}  // namespace p4a
