// router_exact.cuh -- the router in the reference's arithmetic, by one warp. One logit (matvec, src/ref.cpp:68-77: products
// in double, summed in index order, rounded to float once): k_router_pairs (router_gemm.cu) and the routing of decode calls
// (route_block.cuh). Softmax and top-k of one token (src/ref.cpp:574-588): that routing and k_router_topk (route.cu).
#pragma once
#include "common.cuh"

namespace b200moe {

// sp: 256 doubles of shared memory of this warp, or null: NaN where they would be needed. The result is in every lane.
__device__ __forceinline__ float exact_logit(const uint16_t* __restrict__ xr, const uint16_t* __restrict__ wr, int d, double* sp, int lane) {
  double acc = 0, mag = 0;
#pragma unroll 4
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
    if (sp == nullptr) return __int_as_float(0x7fc00000);
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

__device__ __forceinline__ double shfl_f64(double v, int src) {
  return __hiloint2double(__shfl_sync(0xffffffffu, __double2hiint(v), src), __shfl_sync(0xffffffffu, __double2loint(v), src));
}

// Router for one token by one warp, E <= 512: lane holds experts lane, lane+32, ... The reference's arithmetic, out
// of line: only tokens whose ids the logits' order does not decide come here. Weight and id of the lane-th largest.
static __device__ __noinline__ float2 router_one_token(const float* lg, int E, int k, int lane) {
  float v[16];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    int e = j * 32 + lane;
    v[j] = e < E ? lg[e] : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const double dmx = (double)mx;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    int e = j * 32 + lane;
    float p = e < E ? (float)exp((double)v[j] - dmx) : 0.f;
    v[j] = p;
  }
  // Sum of the exponentials, as the reference takes it: in double, in index order. All terms
  // are floats in (0, 1]: when the smallest non-zero one's last mantissa bit still fits a
  // double that holds the total, every partial sum of ANY order is exact, so the tree sum has
  // the very same bits and the E dependent additions are only needed otherwise.
  double se = 0;
  float mn = 2.f;
#pragma unroll
  for (int j = 0; j < 16; j++)
    if (j * 32 + lane < E) {
      se += (double)v[j];
      if (v[j] > 0.f) mn = fminf(mn, v[j]);
    }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    se += __hiloint2double(__shfl_xor_sync(0xffffffffu, __double2hiint(se), o),
                           __shfl_xor_sync(0xffffffffu, __double2loint(se), o));
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  se = shfl_f64(se, 0);  // (inexact sums may differ between lanes in the last bit: take one)
  {
    const int e_min = (int)((__float_as_uint(mn) >> 23) & 0xFF) - 127;
    const int bits_total = (int)((__double2hiint(se) >> 20) & 0x7FF) - 1023 + 2;  // generous by one bit
    const bool exact = mn >= 1.17549435e-38f && bits_total - (e_min - 23) <= 53;
    if (!exact) {  // warp-uniform: mn and se are the same in every lane
      se = 0;  // index order, as the reference sums (zeros change nothing)
#pragma unroll
      for (int j = 0; j < 16; j++)
#pragma unroll 1
        for (unsigned m = __ballot_sync(0xffffffffu, v[j] != 0.f); m; m &= m - 1) se += (double)__shfl_sync(0xffffffffu, v[j], __ffs(m) - 1);
    }
  }
#pragma unroll
  for (int j = 0; j < 16; j++) {
    int e = j * 32 + lane;
    v[j] = e < E ? (float)((double)v[j] / se) : -1.f;
  }
  int my_id = 0;
  float my_p = 0.f;
  double kept = 0;
  for (int r = 0; r < k; r++) {
    // The search starts from an id inside [0, E) (the reference's GPU router starts at `lane`,
    // src/gpu/parts/20_kernels_gemv.inc:1517): with a non-finite logit every probability is NaN, no
    // comparison below is ever true, and the ids written are then still valid expert numbers
    // (with NaN weights, so the token's output is NaN) instead of an out-of-range value.
    float bv = -1.f;
    int bi = min(lane, E - 1);
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (v[j] > bv) {
        bv = v[j];
        bi = j * 32 + lane;
      }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) {
        bv = ov;
        bi = oi;
      }
    }
    bi = __shfl_sync(0xffffffffu, bi, 0);  // (NaN probabilities: the lanes may disagree; take lane 0's)
    bv = __shfl_sync(0xffffffffu, bv, 0);
    if (bv < 0.f) bv = __int_as_float(0x7fc00000);  // nothing was selectable: the weight is NaN, as in the reference
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (j == (bi >> 5) && lane == (bi & 31)) v[j] = -1.f;
    if (lane == r) {
      my_id = bi;
      my_p = bv;
    }
    kept += (double)bv;
  }
  return make_float2((float)((double)my_p / kept), __int_as_float(my_id));
}

}  // namespace b200moe
