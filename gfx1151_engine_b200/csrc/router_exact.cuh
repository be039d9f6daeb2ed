// router_exact.cuh -- one router logit in the reference's arithmetic (matvec, src/ref.cpp:68-77: products in
// double, summed in index order, rounded to float once), by one warp. Used by k_router_pairs (router_gemm.cu)
// and by the routing of decode calls (route_tokens.cu).
#pragma once
#include "common.cuh"

namespace b200moe {

// sp: 256 doubles of shared memory of this warp. The result is in every lane.
__device__ __forceinline__ float exact_logit(const uint16_t* __restrict__ xr, const uint16_t* __restrict__ wr, int d, double* sp, int lane) {
  double acc = 0, mag = 0;
  for (int c = lane * 8; c < d; c += 256) {
    const uint4 xv = *(const uint4*)(xr + c), wv = __ldg((const uint4*)(wr + c));
    const uint16_t* xb = (const uint16_t*)&xv;
    const uint16_t* wb = (const uint16_t*)&wv;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const double pd = (double)bf16_bits_to_f32(wb[j]) * (double)bf16_bits_to_f32(xb[j]);  // exact
      acc += pd;
      mag += fabs(pd);
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    acc += __hiloint2double(__shfl_xor_sync(0xffffffffu, __double2hiint(acc), o),
                            __shfl_xor_sync(0xffffffffu, __double2loint(acc), o));
    mag += __hiloint2double(__shfl_xor_sync(0xffffffffu, __double2hiint(mag), o),
                            __shfl_xor_sync(0xffffffffu, __double2loint(mag), o));
  }
  acc = __hiloint2double(__shfl_sync(0xffffffffu, __double2hiint(acc), 0), __shfl_sync(0xffffffffu, __double2loint(acc), 0));
  mag = __hiloint2double(__shfl_sync(0xffffffffu, __double2hiint(mag), 0), __shfl_sync(0xffffffffu, __double2loint(mag), 0));
  // |index-order sum - true sum| <= gamma(d-1) * sum|p|, |this tree sum - true sum| <=
  // gamma(d/32 + 5) * sum|p| (d/32 additions per lane, five shuffle levels), gamma(n) ~ n * 2^-53;
  // `mag` is within the same tiny factor of sum|p|: 1 % of slack covers both second-order terms
  const double delta = 1.01 * (double)(d + d / 32 + 8) * 1.1102230246251565e-16 * mag;
  if ((float)(acc - delta) != (float)(acc + delta)) {  // warp-uniform
    // replay of the reference's order: the lanes form the (exact) products of 256 elements at a
    // time, lane 0 adds them in index order -- the chain of dependent additions is all that is
    // left on one thread
    acc = 0;
    for (int c0 = 0; c0 < d; c0 += 256) {
      const int c = c0 + lane * 8;
      if (c < d) {
        const uint4 xv = *(const uint4*)(xr + c), wv = __ldg((const uint4*)(wr + c));
        const uint16_t* xb = (const uint16_t*)&xv;
        const uint16_t* wb = (const uint16_t*)&wv;
#pragma unroll
        for (int j = 0; j < 8; j++) sp[lane * 8 + j] = (double)bf16_bits_to_f32(wb[j]) * (double)bf16_bits_to_f32(xb[j]);
      }
      __syncwarp();
      if (lane == 0) {
        const int n = min(256, d - c0);
        for (int j = 0; j < n; j++) acc += sp[j];
      }
      __syncwarp();
    }
  }
  return (float)__hiloint2double(__shfl_sync(0xffffffffu, __double2hiint(acc), 0), __shfl_sync(0xffffffffu, __double2loint(acc), 0));
}

}  // namespace b200moe
