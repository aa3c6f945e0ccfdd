// pair_math_check.cu — p4a_test_pair_math: the claims of pair_math.cuh, checked on the
// device for every float of a range. Not used by the library itself.
#include <cuda_runtime.h>

#include <cstring>

#include "../../include/p4a.h"
#include "pair_math.cuh"

namespace p4a {

namespace {

constexpr uint32_t kListed = 1u << 16;
struct Counts {
  unsigned long long roots, recips, unrounded, quotients;
};

// Floats with the bits first .. last-1: roots that are not sqrtf's, reciprocals that are
// not the rounded ones, and the arguments whose root's reciprocal is not (listed).
__global__ void k_check_roots(uint32_t first, uint32_t last, Counts* c, uint32_t* list) {
  unsigned long long roots = 0, recips = 0;
  for (unsigned long long b = first + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b < last;
       b += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((uint32_t)b), s = sqrtf(x), y = -(1.0f / x);
    const Root1 r = root1(x);
    const Root2 p = root2(splat2(x));
    float s0, s1, y0, y1, r0, r1;
    unpack2(p.s, s0, s1);
    unpack2(p.yn, y0, y1);
    unpack2(recip2(splat2(x)), r0, r1);
    if (r.s != s || s0 != s || s1 != s || y0 != r.yn || y1 != r.yn) roots++;
    if (recip1(x) != y || r0 != y || r1 != y) recips++;
    if (r.yn != -(1.0f / s)) {
      const unsigned long long at = atomicAdd(&c->unrounded, 1ull);
      if (at < kListed) list[at] = (uint32_t)b;
    }
  }
  if (roots) atomicAdd(&c->roots, roots);
  if (recips) atomicAdd(&c->recips, recips);
}

// Quotients by the listed arguments' roots, for the 2^23 numerators from `numerator` on.
__global__ void k_check_quotients(uint32_t numerator, Counts* c, const uint32_t* list) {
  const unsigned long long n = (c->unrounded < kListed ? c->unrounded : kListed) << 23;
  unsigned long long wrong = 0;
  for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    const Root1 r = root1(__uint_as_float(list[t >> 23]));
    const float a = __uint_as_float(numerator + (uint32_t)(t & 0x7fffffu)), q = a / r.s;
    float q0, q1;
    unpack2(quot2(splat2(a), splat2(r.s), splat2(r.yn)), q0, q1);
    if (quot1(a, r.s, r.yn) != q || -q0 != q || -q1 != q) wrong++;
  }
  if (wrong) atomicAdd(&c->quotients, wrong);
}

}  // namespace

}  // namespace p4a

using namespace p4a;

extern "C" int p4a_test_pair_math(float lo, float hi, float numerator, uint64_t counts[4]) {
  if (!(lo >= 0x1p-100f && hi > lo && hi <= 0x1p100f && numerator >= 0x1p-101f && numerator <= 0x1p100f) || !counts)
    return P4A_ERR_ARG;
  uint32_t bits[3];
  const float f[3] = {lo, hi, numerator};
  memcpy(bits, f, sizeof(bits));
  Counts h{};
  Counts* c = nullptr;
  uint32_t* list = nullptr;
  cudaStream_t st = nullptr;
  bool ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMalloc((void**)&c, sizeof(Counts)) == cudaSuccess && cudaMalloc((void**)&list, kListed * 4) == cudaSuccess &&
            cudaMemsetAsync(c, 0, sizeof(Counts), st) == cudaSuccess;
  if (ok) {
    k_check_roots<<<148 * 8, 256, 0, st>>>(bits[0], bits[1], c, list);
    k_check_quotients<<<148 * 8, 256, 0, st>>>(bits[2], c, list);
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpyAsync(&h, c, sizeof(h), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
         cudaStreamSynchronize(st) == cudaSuccess;
  }
  if (list) cudaFree(list);
  if (c) cudaFree(c);
  if (st) cudaStreamDestroy(st);
  counts[0] = h.roots;
  counts[1] = h.recips;
  counts[2] = h.unrounded;
  counts[3] = h.quotients;
  return ok ? P4A_OK : P4A_ERR_CUDA;
}
