// Eight bf16 at a time (16-byte accesses), and the end of a launch: shared by the memory-bound kernels.
#pragma once
#include "common.cuh"

extern "C" void pt_count_launches(int n);

namespace pt {

typedef __nv_bfloat16 bf16;

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

}  // namespace pt

static inline int check_launch(int n = 1) {
  pt_count_launches(n);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
