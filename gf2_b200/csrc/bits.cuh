// gf2cuda bit-matrix helpers (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gf2c {

// 32 x 32 bit transpose across a warp: lane c returns bit r = bit c of lane r's
// x.  Per step one shuffle, then a byte permute (distances 16 and 8) or a
// rotate and a select, with the lane's selectors made once.
struct Transpose32 {
  uint32_t p16, p8, m4, m2, m1;
  int r4, r2, r1;
  __device__ __forceinline__ explicit Transpose32(int lane) {
    p16 = lane & 16 ? 0x3276u : 0x5410u;
    p8 = lane & 8 ? 0x3715u : 0x6240u;
    m4 = lane & 4 ? 0xf0f0f0f0u : 0x0f0f0f0fu;
    m2 = lane & 2 ? 0xccccccccu : 0x33333333u;
    m1 = lane & 1 ? 0xaaaaaaaau : 0x55555555u;
    r4 = lane & 4 ? 28 : 4;
    r2 = lane & 2 ? 30 : 2;
    r1 = lane & 1 ? 31 : 1;
  }
  static __device__ __forceinline__ uint32_t step(uint32_t x, int d, int r, uint32_t m) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, d);
    return (x & m) | (__funnelshift_l(y, y, r) & ~m);
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), p16);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), p8);
    x = step(x, 4, r4, m4);
    x = step(x, 2, r2, m2);
    return step(x, 1, r1, m1);
  }
};

}  // namespace gf2c
