// expert_simt.cu -- expert FFN on the CUDA cores: fp32 weights dequantised exactly as the
// reference does, fp32 FMA accumulation. This is the decode / speculative-verify path
// (T <= 16; takes the place of k_q4cp_gemv_gg, k_silu_mul_g and k_q4cp_gemv_gd,
// src/gpu/parts/20_kernels_gemv.inc:1607-1764, and of the GGUF raw-block GEMV,
// src/gpu/parts/26_kernels_moe_gguf.inc:487-939) and, at any T, the slow exact path the
// tensor-core kernels are cross-checked against.
//
// Work decomposition: one block of 128 threads per (run of rows of one expert, m-tile);
// thread r owns output row r of the tile and streams that row's codes, 16 bytes per
// load, 512 contiguous bytes per warp. Rows of the run are processed NT at a time with
// their activations staged in shared memory (every thread reads the same activation
// address: a broadcast).
#include "kernels.h"

namespace b200moe {

namespace {

constexpr int kNT = 8;        // rows (tokens) per pass
constexpr int kPiece = 1024;  // K elements of activations staged at a time

template <int FMT>
struct RowMeta {};

// Per (row, 32-group) dequantisation constants, and the fp32 value of one code.
template <>
struct RowMeta<kQ4CP> {
  float s;
  const float* book;
  __device__ __forceinline__ void load(const uint8_t* meta, int h, const float* bk) {
    s = half_bits_to_f32(((const uint16_t*)meta)[h]);
    book = bk;
  }
  __device__ __forceinline__ float value(int nib, int) const { return __fmul_rn(book[nib], s); }
};
template <>
struct RowMeta<kQ4K> {
  float d1, dm1;
  __device__ __forceinline__ void load(const uint8_t* meta, int h, const float*) {
    const uint8_t* m = meta;
    float d = half_bits_to_f32(*(const uint16_t*)m), dmin = half_bits_to_f32(*(const uint16_t*)(m + 2));
    d1 = __fmul_rn(d, (float)m[4 + 2 * h]);
    dm1 = __fmul_rn(dmin, (float)m[5 + 2 * h]);
  }
  __device__ __forceinline__ float value(int nib, int) const {
    return __fsub_rn(__fmul_rn(d1, (float)nib), dm1);
  }
};
template <>
struct RowMeta<kQ51> {
  float d, m;
  uint32_t qh;
  __device__ __forceinline__ void load(const uint8_t* meta, int h, const float*) {
    const uint8_t* p = meta + h * 8;
    d = half_bits_to_f32(*(const uint16_t*)p);
    m = half_bits_to_f32(*(const uint16_t*)(p + 2));
    qh = *(const uint32_t*)(p + 4);
  }
  __device__ __forceinline__ float value(int nib, int j) const {
    int x = nib | (int)(fifth_bit_of(qh, j) << 4);
    return __fadd_rn(__fmul_rn((float)x, d), m);
  }
};

constexpr int kQ80 = 3;  // here only: a two-plane image of 8-bit codes (GGUF Q8_0), its planes put together again

// acc[j] += sum over the K range [k0, k0+klen) of w[r][k] * xs[j][k - k0], j < NT
template <int FMT, int NT>
__device__ __forceinline__ void row_dot(const Image& img, int e, int mt, int r, int k0, int klen, const float* book,
                                        const float (*xs)[kPiece], float* acc) {
  for (int kb = k0 / kTileK; kb < (k0 + klen) / kTileK; kb++) {
    const uint8_t *codes = img.codes(e, mt, kb, r), *meta = img.meta(e, mt, kb, r);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint4 c4 = *(const uint4*)(codes + h * kHalfBytes);
      RowMeta<FMT> rm;
      rm.load(meta, h, book);
      const uint32_t wds[4] = {c4.x, c4.y, c4.z, c4.w};
      const int xo = kb * kTileK - k0 + h * 32;
#pragma unroll
      for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int n = 0; n < 8; n++) {
          const int j = q * 8 + n;
          const float w = rm.value((wds[q] >> (4 * n)) & 15, j);
#pragma unroll
          for (int t = 0; t < NT; t++) acc[t] = fmaf(w, xs[t][xo + j], acc[t]);
        }
      }
    }
  }
}

// The 8-bit codes: (16 hi + lo) - 128 is the source's int8 q, put together four at a time; one byte permute makes 2^15 + 128 + q of it and
// one multiply-add d * q, exactly (the scale has 11 bits, 2^15 + 128 nine), so that a sum overflows only where its terms d * q * x do: 3.6
// instructions a weight and one per row, where plane by plane and with the rows' number unknown to the compiler it took about 40. Bound by the HBM then: 9 tokens on 512 experts of
// 4096 x 1024 2037 -> 271 us (5.9 TB/s), one token 570 -> 95; 13 tokens on 512 of 2560 x 640 1166 -> 183.
template <int NT>
__device__ __forceinline__ void row_dot_q80(const Image& img, int e, int mt, int r, int k0, int klen, const float (*xs)[kPiece],
                                            float* acc) {
  struct Block {
    uint4 hi[2], lo[2];
    uint32_t d[2];
  };
  const uint8_t* p = img.codes(e, mt, (k0 / kTileK) * 2, r);  // high plane's K block; the low plane's follows
  constexpr int sub_b = sub_bytes(kQ51);
  const int off_m = meta_offset(kQ51, tile_pos(r, img.paired)) - code_offset(tile_pos(r, img.paired));
  auto load = [&](Block& b) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      b.hi[h] = __ldg((const uint4*)(p + h * kHalfBytes));
      b.lo[h] = __ldg((const uint4*)(p + sub_b + h * kHalfBytes));
      b.d[h] = __ldg((const uint32_t*)(p + sub_b + off_m + h * 8));
    }
    p += 2 * sub_b;
  };
  const int n = klen / kTileK;
  Block b;
  load(b);
  for (int i = 0; i < n; i++) {
    const Block now = b;
    if (i + 1 < n) load(b);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t hi[4] = {now.hi[h].x, now.hi[h].y, now.hi[h].z, now.hi[h].w};
      const uint32_t lo[4] = {now.lo[h].x, now.lo[h].y, now.lo[h].z, now.lo[h].w};
      const float d = half_bits_to_f32((uint16_t)(now.d[h] & 0xFFFFu)), bias = -32896.f * d;
      float sum[NT];
#pragma unroll
      for (int t = 0; t < NT; t++) sum[t] = 0.f;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t even = (lo[q] & 0x0F0F0F0Fu) | ((hi[q] << 4) & 0xF0F0F0F0u), odd = ((lo[q] >> 4) & 0x0F0F0F0Fu) | (hi[q] & 0xF0F0F0F0u);
#pragma unroll
        for (int c = 0; c < 8; c += 4) {
          float w[4];
#pragma unroll
          for (int k = 0; k < 4; k++)
            w[k] = fmaf(__uint_as_float(__byte_perm(k & 1 ? odd : even, 0x47000000u, 0x7504u | (uint32_t)((c + k) >> 1) << 4)), d, bias);
#pragma unroll
          for (int t = 0; t < NT; t++) {
            const float4 v = *(const float4*)&xs[t][i * kTileK + h * 32 + q * 8 + c];
            sum[t] = fmaf(w[3], v.w, fmaf(w[2], v.z, fmaf(w[1], v.y, fmaf(w[0], v.x, sum[t]))));
          }
        }
      }
#pragma unroll
      for (int t = 0; t < NT; t++) acc[t] += sum[t];
    }
  }
}

// nt <= kNT rows: the loops above know 1, 2, 4 or 8 (rows that are not there are computed on what the buffer holds, and dropped)
template <int FMT>
__device__ __forceinline__ void rows_dot(const Image& img, int e, int mt, int r, int k0, int klen, const float* book,
                                         const float (*xs)[kPiece], int nt, float* acc) {
#define B200MOE_ROWS(n)                                                             \
  do {                                                                              \
    if constexpr (FMT == kQ80) row_dot_q80<n>(img, e, mt, r, k0, klen, xs, acc);    \
    else row_dot<FMT, n>(img, e, mt, r, k0, klen, book, xs, acc);                   \
  } while (0)
  if (nt == 1) B200MOE_ROWS(1);
  else if (nt == 2) B200MOE_ROWS(2);
  else if (nt <= 4) B200MOE_ROWS(4);
  else B200MOE_ROWS(8);
#undef B200MOE_ROWS
}

template <int FMT>
__global__ void __launch_bounds__(128)
k_up_simt(Image img, const uint16_t* __restrict__ x, int d, int mid,
          const int32_t* __restrict__ tokidx, const Run* __restrict__ runs,
          const int32_t* __restrict__ n_runs, float* __restrict__ hid) {
  if ((int)blockIdx.y >= *n_runs) return;
  __shared__ __align__(16) float xs[kNT][kPiece];
  __shared__ float us[kNT][64];
  __shared__ float book_s[32];
  const Run run = runs[blockIdx.y];
  const int mt = blockIdx.x, r = threadIdx.x;
  if (r < 32) book_s[r] = img.book ? img.book[r] : 0.f;
  const float* book = book_s + (r >= 64 ? 16 : 0);
  for (int c0 = 0; c0 < run.count; c0 += kNT) {
    const int nt = min(kNT, run.count - c0);
    float acc[kNT];
#pragma unroll
    for (int t = 0; t < kNT; t++) acc[t] = 0.f;
    for (int k0 = 0; k0 < d; k0 += kPiece) {
      const int klen = min(kPiece, d - k0);
      __syncthreads();
      for (int t = 0; t < nt; t++) {
        const uint16_t* row = x + (size_t)tokidx[run.first + c0 + t] * d + k0;
        for (int i = r; i < klen; i += 128) xs[t][i] = bf16_bits_to_f32(row[i]);
      }
      __syncthreads();
      rows_dot<FMT>(img, run.expert, mt, r, k0, klen, book, xs, nt, acc);
    }
    __syncthreads();
    if (r >= 64)
      for (int t = 0; t < nt; t++) us[t][r - 64] = acc[t];
    __syncthreads();
    if (r < 64)
      for (int t = 0; t < nt; t++)
        hid[(size_t)(run.first + c0 + t) * mid + mt * 64 + r] = silu_f32(acc[t]) * us[t][r];
  }
}

template <int FMT>
__global__ void __launch_bounds__(128)
k_down_simt(Image img, const float* __restrict__ hid, int d, int mid, const Run* __restrict__ runs,
            const int32_t* __restrict__ n_runs, float* __restrict__ pairs) {
  if ((int)blockIdx.y >= *n_runs) return;
  __shared__ __align__(16) float xs[kNT][kPiece];
  __shared__ float book_s[32];
  const Run run = runs[blockIdx.y];
  const int mt = blockIdx.x, r = threadIdx.x;
  if (r < 32) book_s[r] = img.book ? img.book[r] : 0.f;
  const float* book = book_s + (r >= 64 ? 16 : 0);
  for (int c0 = 0; c0 < run.count; c0 += kNT) {
    const int nt = min(kNT, run.count - c0);
    float acc[kNT];
#pragma unroll
    for (int t = 0; t < kNT; t++) acc[t] = 0.f;
    for (int k0 = 0; k0 < mid; k0 += kPiece) {
      const int klen = min(kPiece, mid - k0);
      __syncthreads();
      for (int t = 0; t < nt; t++) {
        const float* row = hid + (size_t)(run.first + c0 + t) * mid + k0;
        for (int i = r; i < klen; i += 128) xs[t][i] = row[i];
      }
      __syncthreads();
      rows_dot<FMT>(img, run.expert, mt, r, k0, klen, book, xs, nt, acc);
    }
    for (int t = 0; t < nt; t++) pairs[(size_t)(run.first + c0 + t) * d + mt * 128 + r] = acc[t];
  }
}

}  // namespace

cudaError_t launch_up_simt(const Image& img, const void* x_bf16, int d, int mid,
                           const int32_t* tokidx, const Run* runs, const int32_t* n_runs,
                           int max_runs, float* hid_f32, cudaStream_t st) {
  dim3 grid(img.n_mtiles, max_runs);
  const uint16_t* x = (const uint16_t*)x_bf16;
  if (img.fmt == kQ4CP)
    k_up_simt<kQ4CP><<<grid, 128, 0, st>>>(img, x, d, mid, tokidx, runs, n_runs, hid_f32);
  else if (img.fmt == kQ4K)
    k_up_simt<kQ4K><<<grid, 128, 0, st>>>(img, x, d, mid, tokidx, runs, n_runs, hid_f32);
  else if (img.act_shift)
    k_up_simt<kQ80><<<grid, 128, 0, st>>>(img, x, d, mid, tokidx, runs, n_runs, hid_f32);
  else
    k_up_simt<kQ51><<<grid, 128, 0, st>>>(img, x, d, mid, tokidx, runs, n_runs, hid_f32);
  return cudaGetLastError();
}

cudaError_t launch_down_simt(const Image& img, const float* hid_f32, int d, int mid, const Run* runs,
                             const int32_t* n_runs, int max_runs, float* pairs_f32,
                             cudaStream_t st) {
  dim3 grid(img.n_mtiles, max_runs);
  if (img.fmt == kQ4CP)
    k_down_simt<kQ4CP><<<grid, 128, 0, st>>>(img, hid_f32, d, mid, runs, n_runs, pairs_f32);
  else if (img.fmt == kQ4K)
    k_down_simt<kQ4K><<<grid, 128, 0, st>>>(img, hid_f32, d, mid, runs, n_runs, pairs_f32);
  else if (img.act_shift)
    k_down_simt<kQ80><<<grid, 128, 0, st>>>(img, hid_f32, d, mid, runs, n_runs, pairs_f32);
  else
    k_down_simt<kQ51><<<grid, 128, 0, st>>>(img, hid_f32, d, mid, runs, n_runs, pairs_f32);
  return cudaGetLastError();
}

}  // namespace b200moe
