// Compares the sum-product kernel's division with __fdiv_rn for every operand
// pair that one of its call sites can form (tests/test_gpu_spa_division.py).
#include "spa_math.cuh"

using namespace gf2c;

// Operands of call site `site` for the value x it computes them from.
__device__ bool operands(int site, float x, float& a, float& b) {
  switch (site) {
    case 0: a = x; b = __fadd_rn(2.0f, -x); return true;                     // tanh: x = -expm1
    case 1: a = __fmul_rn(2.0f, x); b = __fsub_rn(1.0f, x); return true;     // atanh: x = the product
    case 2: a = fabsf(__fsub_rn(x, 1.0f)); b = __fadd_rn(x, 1.0f); return true;  // log: x = the significand
    default: {                                                               // log1p: x = y
      const float u = __fadd_rn(1.0f, x);
      a = x;
      b = __fsub_rn(u, 1.0f);
      return u != 1.0f;
    }
  }
}

__global__ void check(int site, unsigned first, unsigned last, unsigned long long* out) {
  unsigned long long bad = 0, tried = 0;
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = first + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i <= last; i += step) {
    float a, b;
    if (!operands(site, __uint_as_float((unsigned)i), a, b)) continue;
    tried++;
    bad += __float_as_uint(div_cr(a, b)) != __float_as_uint(__fdiv_rn(a, b));
  }
  atomicAdd(&out[0], tried);
  atomicAdd(&out[1], bad);
}

// out: {pairs tried, pairs that differ}; x runs over the floats with bits first .. last.
extern "C" int spa_division_check(int site, unsigned first, unsigned last, unsigned long long* out) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 16);
  if (e == cudaSuccess) e = cudaMemset(d, 0, 16);
  if (e == cudaSuccess) {
    check<<<1184, 256>>>(site, first, last, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}

extern "C" float spa_product_max() { return GF2C_SPA_PMAX; }
