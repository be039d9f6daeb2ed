// rotate.cu -- the Hadamard steps of hgn v2 "i4r" experts (dtype 23: 4-bit codes nib - 8, one fp16
// scale per 128 columns, stored in a rotated domain). The reference keeps the weights rotated and
// moves the rotation onto the activations (src/gpu/parts/28_kernels_hgn_v2.inc:1-15):
//   W = diag(svh) . Hn . G . Hn . diag(suh),  Hn = H128 / sqrt(128) block-diagonal, H128 the
//   Sylvester Hadamard matrix in natural order,
// so   y = W x = svh * Hn( G . Hn(suh * x) ).
// One MoE layer therefore is (src/gpu/parts/40_model.inc:4559-4680):
//   xr  = Hn(suh_gu * x)                         k_rot_in     (k_v2_rot of the reference)
//   z   = G_gate_up . xr                         grouped GEMM, no activation function
//   g|u = svh_gu * Hn(z);  h = silu(g) * u;  hr = Hn(suh_dn * h)      k_i4r_mid
//   p   = G_down . hr                            grouped GEMM
//   out = svh_dn * Hn(sum_k w_k p_k)             the combine kernel with its rotation step
// A warp owns one 128-vector: lane l holds elements 4l .. 4l+3, so loads and stores are
// contiguous; index bits 0-1 are butterflies inside the lane, bits 2-6 are lane shuffles. The
// transform in natural order does not depend on the order in which the seven bits are taken.
#include "kernels.h"

namespace b200moe {

namespace {

constexpr float kRs128 = 0.08838834764831845f;  // 1 / sqrt(128)

// in-place 128-point Walsh-Hadamard transform (natural order, unnormalised) of the warp's vector
__device__ __forceinline__ void fwht128(float (&v)[4], int lane) {
  float a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
  v[0] = a + c;
  v[1] = b + d;
  v[2] = a - c;
  v[3] = b - d;
#pragma unroll
  for (int bit = 1; bit < 32; bit <<= 1) {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float o = __shfl_xor_sync(0xffffffffu, v[j], bit);
      v[j] = upper ? o - v[j] : v[j] + o;
    }
  }
}

__device__ __forceinline__ uint32_t pack_f16x2_sat(float lo, float hi) {
  uint32_t r;  // finite values saturate to the fp16 range, NaN stays NaN
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// x_sorted[row][b*128 ..] = fp16( Hn(pre * x[t][b*128 ..]) ) for the k rows of token t (pairids; negative:
// dropped by the bucketing), one warp per (token, block): rotated once, written k times, no rotated
// copy in token order in between
__global__ void __launch_bounds__(256)
k_rot_in(const uint16_t* __restrict__ x, const float* __restrict__ pre, const int32_t* __restrict__ pairids, int T, int k,
         int d, __half* __restrict__ x_sorted) {
  const int lane = threadIdx.x & 31;
  const int nb = d >> 7;
  pdl_trigger();
  pdl_wait();
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)T * nb) return;
  const int t = (int)(w / nb), b = (int)(w % nb);
  const size_t off = (size_t)t * d + b * 128 + lane * 4;
  const uint2 u = *(const uint2*)(x + off);
  const float4 p = *(const float4*)(pre + b * 128 + lane * 4);
  float v[4] = {bf16_bits_to_f32((uint16_t)(u.x & 0xFFFFu)) * p.x, bf16_bits_to_f32((uint16_t)(u.x >> 16)) * p.y,
                bf16_bits_to_f32((uint16_t)(u.y & 0xFFFFu)) * p.z, bf16_bits_to_f32((uint16_t)(u.y >> 16)) * p.w};
  fwht128(v, lane);
  uint2 o;
  o.x = pack_f16x2_sat(v[0] * kRs128, v[1] * kRs128);
  o.y = pack_f16x2_sat(v[2] * kRs128, v[3] * kRs128);
  for (int s = 0; s < k; s++) {
    const int row = pairids[(size_t)t * k + s];
    if (row >= 0) *(uint2*)(x_sorted + (size_t)row * d + b * 128 + lane * 4) = o;
  }
}

__device__ __forceinline__ void load8(const __half* p, float* v) {
  const uint4 u = *(const uint4*)p;
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __half22float2(*(const __half2*)&w[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

// The same transform by eight lanes: lane l holds elements 8l .. 8l+7 and 64+8l .. 64+8l+7, so index bits 0-2 and 6 are
// butterflies inside the lane and bits 3-5 lane shuffles: 12 a vector and warp, against 20 with a vector per warp.
__device__ __forceinline__ void fwht128_8(float (&v)[16], int lane) {
#pragma unroll
  for (int b = 1; b < 16; b <<= 1)
#pragma unroll
    for (int i = 0; i < 16; i++)
      if (!(i & b)) {
        const float p = v[i], q = v[i | b];
        v[i] = p + q;
        v[i | b] = p - q;
      }
#pragma unroll
  for (int bit = 1; bit < 8; bit <<= 1) {
    const float sign = (lane & bit) ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = fmaf(sign, v[i], __shfl_xor_sync(0xffffffffu, v[i], bit));
  }
}

// hr[row][b*128 ..] = fp16( Hn( suh_dn * silu(g) * u ) ) with g = svh_gu * Hn(z[row][b*128 ..]),
// u = svh_gu[mid + ..] * Hn(z[row][mid + b*128 ..]) (k_i4r_mid of the reference,
// src/gpu/parts/28_kernels_hgn_v2.inc:98-143). Eight lanes per (row, block b = blockIdx.y of mid), whose planes stay in
// registers. With a warp per vector, 60 shuffles and 64-bit index arithmetic bounded it, not its 6 bytes a hidden
// value: 20480 rows of 640 took 45 us (78 MB: 12 us at the copy bandwidth). Of a whole 2048-token call (724 us) the
// gain is below what two runs differ by.
__global__ void __launch_bounds__(256)
k_i4r_mid(const __half* __restrict__ z, const float* __restrict__ svh_gu, const float* __restrict__ suh_dn,
          int rows, int mid, __half* __restrict__ hr) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.y * 128 + (lane & 7) * 8;
  float sg[16], su[16], sd[16];
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int e = c + (i & 7) + (i >> 3) * 64;
    sg[i] = svh_gu[e];
    su[i] = svh_gu[mid + e];
    sd[i] = suh_dn[e];
  }
  pdl_trigger();
  pdl_wait();
  // (whole warps stay in the loop: the shuffles take all lanes)
  for (int r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 4; r0 < rows; r0 += gridDim.x * 32) {
    const int row = r0 + (lane >> 3);
    const bool live = row < rows;
    float g[16], u[16];
    const __half* zr = z + (size_t)(live ? row : r0) * 2 * mid + c;
    load8(zr, g);
    load8(zr + 64, g + 8);
    load8(zr + mid, u);
    load8(zr + mid + 64, u + 8);
    fwht128_8(g, lane);
    fwht128_8(u, lane);
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const float gv = g[i] * kRs128 * sg[i], uv = u[i] * kRs128 * su[i];
      g[i] = silu_f32(gv) * uv * sd[i];
    }
    fwht128_8(g, lane);
    if (!live) continue;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint4 o;
      o.x = pack_f16x2_sat(g[8 * h] * kRs128, g[8 * h + 1] * kRs128);
      o.y = pack_f16x2_sat(g[8 * h + 2] * kRs128, g[8 * h + 3] * kRs128);
      o.z = pack_f16x2_sat(g[8 * h + 4] * kRs128, g[8 * h + 5] * kRs128);
      o.w = pack_f16x2_sat(g[8 * h + 6] * kRs128, g[8 * h + 7] * kRs128);
      *(uint4*)(hr + (size_t)row * mid + c + h * 64) = o;
    }
  }
}

__global__ void k_f16_to_f32(const uint16_t* __restrict__ src, float* __restrict__ dst, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = half_bits_to_f32(src[i]);
}

}  // namespace

cudaError_t launch_rot_in(const void* x_bf16, const float* pre, const int32_t* pairids, int T, int k, int d,
                          __half* x_sorted, cudaStream_t st) {
  const long long warps = (long long)T * (d >> 7);
  if (warps == 0) return cudaSuccess;
  return launch_pdl(k_rot_in, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, st, (const uint16_t*)x_bf16, pre, pairids, T, k, d,
                    x_sorted);
}

cudaError_t launch_i4r_mid(const __half* z, const float* svh_gu, const float* suh_dn, int rows, int mid, __half* hr,
                           cudaStream_t st) {
  const int nb = mid >> 7, per_wave = 148 * 4;  // blocks of 32 rows a wave takes (registers: two a SM, two waves)
  int gx = (rows + 31) / 32;
  if ((long long)gx * nb > per_wave) gx = (per_wave + nb - 1) / nb;
  if (gx < 1) gx = 1;
  return launch_pdl(k_i4r_mid, dim3((unsigned)gx, (unsigned)nb), dim3(256), 0, st, z, svh_gu, suh_dn, rows, mid, hr);
}

cudaError_t launch_f16_to_f32(const void* src_f16_dev, float* dst, int n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_f16_to_f32<<<(n + 255) / 256, 256, 0, st>>>((const uint16_t*)src_f16_dev, dst, n);
  return cudaGetLastError();
}

}  // namespace b200moe
