// The packed operations of f32x2.cuh beside the scalar ones, for
// test_gpu_f32x2.py: out[0..n) div2, [n..2n) __fdiv_rn, then mul2 and
// __fmul_rn, then add2(mul2(a, b), c) and the separately rounded sum.
#include "f32x2.cuh"
#include "shb_internal.h"

namespace {
__global__ void k_probe(const float* a, const float* b, const float* c, int64_t n, float* out) {
  using namespace shb;
  for (int64_t i = 2 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); i + 1 < n;
       i += 2 * (int64_t)gridDim.x * blockDim.x) {
    const float a0 = a[i], a1 = a[i + 1], b0 = b[i], b1 = b[i + 1], c0 = c[i], c1 = c[i + 1];
    const f32x2 av = pack2(a0, a1), bv = pack2(b0, b1);
    const float2 q = unpack2(div2(av, pack2(-b0, -b1), pack2(__frcp_rn(b0), __frcp_rn(b1))));
    const float2 m = unpack2(mul2(av, bv)), s = unpack2(add2(mul2(av, bv), pack2(c0, c1)));
    const float want[6] = {__fdiv_rn(a0, b0), __fdiv_rn(a1, b1), __fmul_rn(a0, b0), __fmul_rn(a1, b1),
                           __fadd_rn(__fmul_rn(a0, b0), c0), __fadd_rn(__fmul_rn(a1, b1), c1)};
    const float got[6] = {q.x, q.y, m.x, m.y, s.x, s.y};
    for (int k = 0; k < 3; ++k)
      for (int h = 0; h < 2; ++h) {
        out[2 * k * n + i + h] = got[2 * k + h];
        out[(2 * k + 1) * n + i + h] = want[2 * k + h];
      }
  }
}
}  // namespace

// n even, all pointers on the current device, out 6 n floats.
extern "C" __attribute__((visibility("default"))) int f32x2_probe(const float* a, const float* b, const float* c,
                                                                  int64_t n, float* out) {
  k_probe<<<592, 256>>>(a, b, c, n, out);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

// The range that lights weighed in pairs are held to.
extern "C" __attribute__((visibility("default"))) void f32x2_range(float r[4]) {
  r[0] = shb::kPairDim, r[1] = shb::kPairBright, r[2] = shb::kPairNear, r[3] = shb::kPairFar;
}
