// tc.h -- interface of the tcgen05 grouped dequant-GEMM (expert_tc.cu).
#pragma once
#include "common.cuh"

namespace b200moe {

struct TcPlan;  // tensor maps over the activation buffers + device properties

// x_sorted: [rows_cap][d] fp16 (expert-sorted activations); hid16: [rows_cap][mid] fp16.
cudaError_t tc_create(TcPlan** plan, const __half* x_sorted, const __half* hid16,
                      long long rows_cap, int d, int mid);
void tc_destroy(TcPlan* plan);
// expert_dense.cu: the down GEMM of popular experts. w: where the expanded weights of `cap` experts go, [cap][d][mid] fp16.
cudaError_t tc_set_dense(TcPlan* plan, const __half* w, int cap, int d, int mid);
cudaError_t launch_expand(const TcPlan* plan, const Image& img, const int32_t* experts, const int32_t* n_dense, __half* out,
                          cudaStream_t st);
cudaError_t launch_down_dense(const TcPlan* plan, const Tile* tiles, const int32_t* n_dense, int d, int mid, __half* pairs16, int32_t* status,
                              cudaStream_t st);
// Leave `sms` SMs free of the persistent GEMM CTAs (for communication kernels that must run
// at the same time). The two launches above are refused on such a plan.
void tc_set_sm_margin(TcPlan* plan, int sms);

// Largest number of rows in one grouped-GEMM tile (the MMA N extent), and in one of a narrow launch.
constexpr int kTcTileN = 192;
constexpr int kTcNarrowN = 64;

struct TcLaunch {
  bool narrow = false;  // every tile of the list has at most kTcNarrowN rows
  // The launch may run at the same time as the one in front of it in the stream, which must be another
  // of these launches (either form), the popular experts' GEMM or the decode GEMV's, on other rows; it is complete only when that one is.
  bool beside = false;
  // down GEMM; rowmap + map_base (device, both or neither): result row r >= map_base[0] of the tile list goes
  // to pairs16[rowmap[r - map_base[0]]] instead of pairs16[r].
  const int32_t* rowmap = nullptr;
  const int32_t* map_base = nullptr;
  const int32_t* skip = nullptr;  // device: so many tiles of the list, the first, are not this launch's (wide form)
};

// gate/up GEMM + SwiGLU: hid16[row][mid] = silu(W_gate x) * (W_up x) for every row of every tile.
cudaError_t launch_up_tc(TcPlan* plan, const Image& img, const Tile* tiles, const int32_t* n_tiles,
                         int max_tiles, __half* hid16, int32_t* status, cudaStream_t st, const TcLaunch& o = {});
// down GEMM: pairs16[row][d] = W_down hid16[row].
cudaError_t launch_down_tc(TcPlan* plan, const Image& img, const Tile* tiles, const int32_t* n_tiles,
                           int max_tiles, __half* pairs16, int32_t* status, cudaStream_t st, const TcLaunch& o = {});

// expert_few.cu: one of these GEMMs with tiles of at most kTcNarrowN rows (up: gate/up + SwiGLU; hidden: of the hidden
// activations, else of x_sorted).
cudaError_t launch_few(const TcPlan* plan, bool up, bool hidden, const Image& img, const Tile* tiles, const int32_t* n_tiles, int max_tiles,
                       __half* out, int out_ld, int32_t* status, cudaStream_t st, bool beside);

// plain GEMM over the expert-sorted activations (no activation function): z16[row][n_mtiles*128] =
// W x_sorted[row], for images whose rows are not gate/up pairs (hgn v2 i4r gate_up).
cudaError_t launch_raw_tc(TcPlan* plan, const Image& img, const Tile* tiles, const int32_t* n_tiles,
                          int max_tiles, __half* z16, int32_t* status, cudaStream_t st, const TcLaunch& o = {});

}  // namespace b200moe
