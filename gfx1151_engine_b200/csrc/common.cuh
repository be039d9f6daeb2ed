// common.cuh -- shared definitions of the B200 MoE operator (tile geometry, device
// helpers, internal structs). Host and device.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200moe {

// ---- repacked weights ---------------------------------------------------------------
// A quantised expert tensor is a grid of tiles of 128 output rows x 64 K elements, a tile four sub-blocks
// of 32 rows. A sub-block is one contiguous object of whole 128-byte lines, {codes of half 0, codes of half 1,
// metadata}: 512 code bytes per half h, 16 per row with the 32 four-bit codes of the row for
// K = 64*kb + 32*h .. +31, low nibble = even K (the nibble order of hgn q4cp, src/hgn.h:5-9 of the reference), then
// the rows' metadata, whose size depends on the source format. A plain image holds rows 32s .. 32s+31 of the
// tile in sub-block s; a paired (gate/up) one gate rows 16s .. 16s+15 and the matching up rows 64+16s .. 64+16s+15.
//   [expert][m_tile][sub-block 0..3][k_block][sub-block bytes]
// The decode GEMV walks 16 hidden outputs (or 32 output rows) along K: one stream, a warp's K blocks one
// bulk copy. A warp of the tensor-core kernel owns the 32 rows of a sub-block (or 16 rows of two): a
// read of its rows of a half touches four whole lines.
constexpr int kTileM = 128;
constexpr int kTileK = 64;
constexpr int kSubRows = 32;
constexpr int kSubCodes = kSubRows * kTileK / 2;  // 1024

enum Format : int {
  kQ4CP = 0,  // metadata of a row: {fp16 scale of half 0, of half 1}
  kQ4K = 1,   // {fp16 d, fp16 dmin, u8 sc0, u8 m0, u8 sc1, u8 m1}
  kQ51 = 2    // {fp16 d0, fp16 m0, u32 fifth bits 0, fp16 d1, fp16 m1, u32 fifth bits 1}
};
// kQ51, the fifth-bit word of a 32-group: bit i (i < 16) belongs to the LOW-nibble code of code
// byte i (element 2i of the group), bit 16 + i to its high-nibble code (element 2i + 1). With the
// two bits of a code byte 16 apart, one shift and one mask move them to bits 14 and 30 -- the
// fp16 pair (2.0 or 0, 2.0 or 0) -- and a single half2 multiply-add by 8 adds the 16s to the two
// looked-up codes.
__host__ __device__ inline uint32_t fifth_bits_split(uint32_t by_element) {  // bit j = element j  ->  the layout above
  uint32_t r = 0;
  for (int i = 0; i < 16; i++)
    r |= (((by_element >> (2 * i)) & 1u) << i) | (((by_element >> (2 * i + 1)) & 1u) << (16 + i));
  return r;
}
__host__ __device__ inline uint32_t fifth_bit_of(uint32_t split, int j) {  // fifth bit of element j of the group
  return (split >> ((j & 1) ? 16 + (j >> 1) : (j >> 1))) & 1u;
}
// GGUF Q8_0 (int8 codes q, fp16 d per 32: w = d * q) has no tile layout of its own. With the
// biased code u = q + 128 = 16 * hi + lo the weight is d * (16 * hi - 128) + d * lo: two 4-bit
// tensors over the SAME activations. The image is kQ51 with twice the K blocks -- for every 64
// columns a block of the high nibbles (group constants d' = 16 d, m' = -128 d, no fifth bits)
// followed by a block of the low nibbles (d' = d, m' = 0) -- and act_shift = 1. 16 d and 128 d are
// exact in fp16, so every kernel reproduces d * q up to its usual single rounding.

__host__ __device__ constexpr int meta_row_bytes(int fmt) { return fmt == kQ4CP ? 4 : fmt == kQ4K ? 8 : 16; }
__host__ __device__ constexpr int sub_bytes(int fmt) { return kSubCodes + kSubRows * meta_row_bytes(fmt); }  // 1152, 1280, 1536
__host__ __device__ constexpr int tile_bytes(int fmt) { return kTileM / kSubRows * sub_bytes(fmt); }
// Where tile row r sits: its sub-block (bits 5 and up) and its place there.
__host__ __device__ constexpr int tile_pos(int r, int paired) {
  return paired ? ((r & 63) >> 4) * kSubRows + (r >> 6) * 16 + (r & 15) : r;
}
// Inside a sub-block: the 16 code bytes of half 0 of the row at place `pos` (half 1 lies kHalfBytes further), its metadata.
constexpr int kHalfBytes = kSubRows * 16;
__host__ __device__ constexpr int code_offset(int pos) { return (pos & 31) * 16; }
__host__ __device__ constexpr int meta_offset(int fmt, int pos) { return kSubCodes + (pos & 31) * meta_row_bytes(fmt); }

// One repacked tensor set: n_experts x n_mtiles x n_kblocks tiles.
struct Image {
  uint8_t* data = nullptr;
  int fmt = kQ4CP;
  int n_experts = 0;
  int n_mtiles = 0;   // per expert
  int n_kblocks = 0;  // K / 64
  int paired = 0;     // 1: gate/up image (tile rows 0..63 gate, 64..127 the matching up rows)
  int dual_book = 0;  // 1: the two halves of a tile use different code books (separate gate / up tensors)
  int act_shift = 0;  // 1: two-plane image of 8-bit codes (GGUF Q8_0): K block kb of the image multiplies the
                      //    activations of K block kb >> 1 -- the high and the low nibble plane of the same 64 columns
  float* book = nullptr;  // device [32]: code book of tile rows 0..63, then of rows 64..127
  __host__ __device__ size_t mtile_stride() const { return (size_t)n_kblocks * tile_bytes(fmt); }
  __host__ __device__ size_t expert_stride() const { return n_mtiles * mtile_stride(); }
  __host__ __device__ uint8_t* mtile(int e, int mt) const { return data + ((size_t)e * n_mtiles + mt) * mtile_stride(); }
  // from mtile(): the sub-block of tile row r in K block 0; the next K block lies sub_bytes(fmt) further
  __host__ __device__ size_t row_sub(int r) const { return (size_t)(tile_pos(r, paired) >> 5) * n_kblocks * sub_bytes(fmt); }
  // codes (half 0) and metadata of a tile row in K block kb
  __host__ __device__ uint8_t* codes(int e, int mt, int kb, int r) const {
    return mtile(e, mt) + row_sub(r) + (size_t)kb * sub_bytes(fmt) + code_offset(tile_pos(r, paired));
  }
  __host__ __device__ uint8_t* meta(int e, int mt, int kb, int r) const {
    return mtile(e, mt) + row_sub(r) + (size_t)kb * sub_bytes(fmt) + meta_offset(fmt, tile_pos(r, paired));
  }
};

// A run of permuted rows that belong to one expert (the unit the expert kernels work on).
struct Run {
  int expert;
  int first;
  int count;
};

// Work item of the grouped GEMM: rows of one expert, at most as many as the launch that reads the list takes
// (kTcTileN, narrow launches kTcNarrowN: whoever writes a list cuts it to that).
struct Tile {
  int expert;
  int first;
  int count;
};

// Rows of a tile of the GEMM on expanded weights (expert_dense.cu), and of the least that is whole tiles both there and in
// the grouped dequant-GEMM (4 of kTcTileN).
constexpr int kDenseRows = 256, kDenseGroup = 768;

constexpr int kMaxTopK = 16;
constexpr int kMaxExperts = 512;
constexpr int kIdStride = 16;  // internal top-k rows are 16 wide, like the engine's

// ---- device helpers ----------------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_f32(uint16_t b) {
  return __uint_as_float((uint32_t)b << 16);
}
__device__ __forceinline__ float half_bits_to_f32(uint16_t h) {
  return __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ float silu_f32(float v) { return v / (1.f + expf(-v)); }
__device__ __forceinline__ float sigmoid_f32(float v) { return 1.f / (1.f + expf(-v)); }

}  // namespace b200moe
