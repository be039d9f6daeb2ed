// route.cu -- router top-k and the expert bucketing of (token, slot) pairs.
//
// Semantics follow the reference:
//   * probabilities as its CPU path forms them (src/ref.cpp:574-582): exp in double of
//     (logit - max), rounded to float, summed in double in index order, divided in
//     double, rounded to float; selection of the k largest, descending, ties to the lowest
//     expert id (the rule of its GPU router, src/gpu/parts/20_kernels_gemv.inc:1488-1494);
//     weights p / sum(selected p) with the sum taken in rank order (src/ref.cpp:587-588, 606).
//   * bucketing = stable sort of pair index p = t*k + s by expert
//     (src/gpu/parts/10_ple_io.inc:844-853; CPU twin src/gpu/parts/40_model.inc:4171-4183),
//     eoff filled for empty experts too, pairids[t*k + rank] with rank = number of the
//     token's experts with a smaller id (src/gpu/parts/10_ple_io.inc:802-806).
// Everything here is integer/bookkeeping work and deterministic: no atomics on global
// memory, no dependence on block scheduling order.
#include "kernels.h"
#include "route_block.cuh"
#include "tc.h"

namespace b200moe {

namespace {

constexpr int kRouterWarps = 8;

constexpr int kChunk = 512;  // pairs handled by one block (a thread per pair) of the bucketing kernels

__global__ void __launch_bounds__(kRouterWarps * 32)
k_router_topk(const float* __restrict__ logits, int T, int E, int k, int32_t* __restrict__ ids,
              float* __restrict__ w, int stride) {
  __shared__ float s_c[kRouterWarps][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * kRouterWarps + warp;
  pdl_trigger();
  pdl_wait();
  if (t >= T) return;
  // The ids from the logits' order where that decides them (route_block.cuh), which saves E double exponentials and
  // divisions and k rounds of arg-max: 16384 tokens x 512 experts 24 us (33.6 MB: 5 us at the copy bandwidth), with them 63;
  // 77 tokens 5 us and 11.
  float vr, wv;
  int id;
  const int C = warp_leaders(logits + (size_t)t * E, E, k, lane, s_c[warp], vr, id);
  if (C > 0 && warp_topk(logits + (size_t)t * E, E, C, vr, k, lane, true, wv)) {
    for (int i = lane; i < stride; i += 32) {  // zeros behind the k
      ids[(size_t)t * stride + i] = i < k ? id : 0;
      w[(size_t)t * stride + i] = i < k ? wv : 0.f;
    }
  } else {
    const float2 r = router_one_token(logits + (size_t)t * E, E, k, lane);
    for (int i = lane; i < stride; i += 32) {
      ids[(size_t)t * stride + i] = i < k ? __float_as_int(r.y) : 0;
      w[(size_t)t * stride + i] = i < k ? r.x : 0.f;
    }
  }
}

// Decode / verify (T <= 16, T*k <= 256): the whole routing stage in one block (route_block.cuh). Warps 0..15 route,
// warps 16..31 form the shared expert's gates.
__global__ void __launch_bounds__(1024)
k_route_block(const __grid_constant__ RouteIn q) {
  extern __shared__ __align__(16) uint8_t rsm[];
  __shared__ uint8_t row_token[kSmallPairs];
  __shared__ double gpart[16 * 16];
  pdl_trigger();
  pdl_wait();  // inputs may come from the previous kernel; the buffers written here may still be read by it
  if (threadIdx.x < 512) {
    route_block(q, *(RouteBlock*)rsm, true, 16, row_token, [](int, int, int, int) {});
  } else if (q.gate_w) {
    gate_block(q, 0, 1, threadIdx.x - 512, gpart, [] { asm volatile("bar.sync 2, 512;" ::: "memory"); });
  }
}

__global__ void __launch_bounds__(kChunk)
k_route_count(const int32_t* __restrict__ ids, int stride, int pairs, int k, int E,
              int32_t* __restrict__ blockcnt, int32_t* __restrict__ status) {
  __shared__ int hist[kMaxExperts];
  pdl_trigger();
  for (int e = threadIdx.x; e < E; e += kChunk) hist[e] = 0;
  pdl_wait();
  __syncthreads();
  const int p = blockIdx.x * kChunk + threadIdx.x;
  if (p < pairs) {
    const int e = ids[(size_t)(p / k) * stride + p % k];
    if ((unsigned)e < (unsigned)E) atomicAdd(&hist[e], 1);  // ids outside [0, E) are dropped, never used as an index
    else if (status && atomicCAS(status, 0, kStatusBadId) == 0) status[1] = e;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kChunk) blockcnt[(size_t)blockIdx.x * E + e] = hist[e];
}

// One block of 512 threads: per-expert exclusive prefix over the chunk counts, expert
// offsets, the list of non-empty experts and the grouped-GEMM tile list (full tiles first,
// then the ragged ones in descending size so that a static round-robin stays balanced).
__global__ void __launch_bounds__(kMaxExperts)
k_route_scan(int32_t* __restrict__ blockcnt, int nblk, int E, int pairs, int T, TileCut cut,
             int32_t* __restrict__ eoff, Run* __restrict__ runs, int32_t* __restrict__ n_runs,
             Tile* __restrict__ tiles, Tile* __restrict__ tiles_narrow, Tile* __restrict__ tiles_sh, int32_t* __restrict__ n_tiles,
             Tile* __restrict__ tiles_dense, int32_t* __restrict__ dense_experts, int32_t* __restrict__ n_dense) {
  __shared__ __align__(4) uint16_t s_bin[kMaxExperts / 32][kTcTileN + 8];  // ragged tiles of a size: per warp, then in the warps before
  __shared__ int s_gt[256], s_gw[8];                          // larger ones, of all
  __shared__ unsigned long long s_w[kMaxExperts / 32];
  __shared__ int s_wc[kMaxExperts / 32], s_sum[3][kMaxExperts / 32];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  pdl_trigger();
  pdl_wait();
  int cnt = 0;
  if (e < E) {
    // exclusive prefix down this expert's column of the chunk counts; the loads of sixteen
    // rows are issued together so that the walk does not pay one memory latency per chunk
    for (int b = 0; b < nblk; b += 16) {
      int c[16];
#pragma unroll
      for (int i = 0; i < 16; i++) c[i] = b + i < nblk ? blockcnt[(size_t)(b + i) * E + e] : 0;
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (b + i < nblk) {
          blockcnt[(size_t)(b + i) * E + e] = cnt;
          cnt += c[i];
        }
    }
  }
  // experts with few rows to the decode GEMV, where there are enough of them
  const bool by_gemv = cut.gemv_rows > 0 && __syncthreads_count(cnt > 0 && cnt <= cut.gemv_rows) >= cut.min_few && cnt <= cut.gemv_rows;
  int tile_cap = cut.routed, narrow = cut.narrow;
  if (narrow > 0) {
    // one list of wide tiles, one of narrow ones, or both: whichever costs least
    const int rows = by_gemv ? 0 : cnt, part = rows % tile_cap;
    const int n[3] = {(rows + tile_cap - 1) / tile_cap, (rows + narrow - 1) / narrow, part > 0 && part <= narrow};
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const int sum = __reduce_add_sync(0xffffffffu, n[i]);
      if (lane == 0) s_sum[i][warp] = sum;
    }
    __syncthreads();
    int all[3] = {0, 0, 0};
#pragma unroll
    for (int w = 0; w < kMaxExperts / 32; w++)
#pragma unroll
      for (int i = 0; i < 3; i++) all[i] += s_sum[i][w];
    const int wide = kTileCostWide * all[0], few = kTileCostFew * all[1];
    const int both = kTileCostWide * (all[0] - all[2]) + kTileCostFew * all[2] + cut.second;
    if (few <= wide && few <= both) tile_cap = narrow;
    else if (wide <= both) narrow = 0;
  }
  // popular experts: what is whole tiles in both GEMMs goes to the one on expanded weights, for the down stage
  int slot = -1, n_groups = 0, groups0 = 0, all_groups = 0;  // place among them; groups, before it, of all
  if (cut.dense_rows > 0 && tile_cap == kTcTileN) {
    const bool popular = cnt >= cut.dense_rows && cnt >= kDenseGroup;
    const unsigned vote = __ballot_sync(0xffffffffu, popular);
    __syncthreads();
    if (lane == 0) s_sum[0][warp] = __popc(vote);
    __syncthreads();
    int before = __popc(vote & ((1u << lane) - 1u));
    for (int w = 0; w < warp; w++) before += s_sum[0][w];
    if (popular && before < cut.dense_cap) {
      slot = before;
      n_groups = cnt / kDenseGroup;
      dense_experts[slot] = e;
    }
    groups0 = n_groups;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, groups0, o);
      if (lane >= o) groups0 += v;
    }
    if (lane == 31) s_sum[1][warp] = groups0;
    groups0 -= n_groups;
    const int n_slots = __syncthreads_count(slot >= 0);
    for (int w = 0; w < kMaxExperts / 32; w++) {
      if (w < warp) groups0 += s_sum[1][w];
      all_groups += s_sum[1][w];
    }
    if (e == 0) {
      n_dense[0] = all_groups * (kDenseGroup / kDenseRows);
      n_dense[1] = n_slots;
      n_dense[2] = all_groups * (kDenseGroup / kTcTileN);
    }
  } else if (cut.dense_rows > 0 && e < 3) {
    n_dense[e] = 0;
  }
  const bool listed = cnt > 0 && (by_gemv || cut.gemv_rows == 0);
  // three inclusive scans side by side: counts (low 32 bits) and non-empty flags, full tiles
  const int in_groups = n_groups * (kDenseGroup / kTcTileN);  // full tiles that stand in front of the others
  const int nfull = by_gemv ? 0 : cnt / tile_cap - in_groups, part = by_gemv ? 0 : cnt % tile_cap;
  unsigned long long ab = (unsigned long long)(uint32_t)cnt | (unsigned long long)listed << 32;
  int c = nfull;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(0xffffffffu, ab, o);
    const int v = __shfl_up_sync(0xffffffffu, c, o);
    if (lane >= o) {
      ab += u;
      c += v;
    }
  }
  if (lane == 31) {
    s_w[warp] = ab;
    s_wc[warp] = c;
  }
  for (int i = e; i < (int)sizeof(s_bin) / 4; i += kMaxExperts) ((uint32_t*)s_bin)[i] = 0;
  __syncthreads();
  const unsigned same = __match_any_sync(0xffffffffu, part);
  if (lane == __ffs(same) - 1) s_bin[warp][part] = (uint16_t)__popc(same);
  __syncthreads();
  // rank of the ragged tile among all ragged tiles: larger first, ties to the lower id (a loop over the 512 sizes took
  // most of this kernel's 17 us on a short prompt)
  const int bin = 255 - e;
  int above = 0;
  if (e < 256) {
    int tot = 0;
    if (bin <= kTcTileN)
#pragma unroll
      for (int w = 0; w < kMaxExperts / 32; w++) {
        const int n = s_bin[w][bin];
        s_bin[w][bin] = (uint16_t)tot;
        tot += n;
      }
    above = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, above, o);
      if (lane >= o) above += v;
    }
    if (lane == 31) s_gw[warp] = above;
    above -= tot;
  }
  __syncthreads();
  if (e < 256) {
    for (int w = 0; w < warp; w++) above += s_gw[w];
    s_gt[bin] = above;
  }
  __syncthreads();
  const int nparts = s_gt[0], wide_parts = s_gt[narrow], rank = s_gt[part] + s_bin[warp][part] + __popc(same & ((1u << lane) - 1u));
  unsigned long long ab_all = 0;
  int c_all = 0;
#pragma unroll
  for (int w = 0; w < kMaxExperts / 32; w++) {
    const unsigned long long u = s_w[w];
    const int v = s_wc[w];
    if (w < warp) {
      ab += u;
      c += v;
    }
    ab_all += u;
    c_all += v;
  }
  const int first = (int)(uint32_t)ab - cnt, total_full = c_all + all_groups * (kDenseGroup / kTcTileN);
  if (e < E) eoff[e] = first;
  if (e == 0) {
    eoff[E] = (int)(uint32_t)ab_all;  // pairs placed (= T*k unless ids outside [0, E) were dropped)
    n_runs[0] = (int)(ab_all >> 32);
    n_runs[1] = 1;  // the shared expert's run, kept at runs[kMaxExperts]
    runs[kMaxExperts] = Run{0, pairs, T};
  }
  if (listed) runs[(int)(ab >> 32) - 1] = Run{e, first, cnt};
  // full tiles first, then the ragged ones from large to small: those with more than `narrow` rows on tiles
  const int n_wide = tile_cap > narrow ? total_full + wide_parts : 0;
  auto put = [&](int i, const Tile& t) {
    if (i < n_wide) tiles[i] = t;
    else tiles_narrow[i - n_wide] = t;
  };
  const int full0 = total_full - c_all + c - nfull;
  for (int j = 0; j < in_groups; j++) put(groups0 * (kDenseGroup / kTcTileN) + j, Tile{e, first + j * tile_cap, tile_cap});
  for (int j = 0; j < n_groups * (kDenseGroup / kDenseRows); j++)
    tiles_dense[groups0 * (kDenseGroup / kDenseRows) + j] = Tile{slot, first + j * kDenseRows, kDenseRows};
  const int rest = first + in_groups * tile_cap;
  for (int j = 0; j < nfull; j++) put(full0 + j, Tile{e, rest + j * tile_cap, tile_cap});
  if (part > 0) put(total_full + rank, Tile{e, rest + nfull * tile_cap, part});
  // tiles of the shared expert: all T tokens in token order, rows behind the routed ones
  const int nsh = (T + cut.shared - 1) / cut.shared;
  for (int j = e; j < nsh; j += kMaxExperts)
    tiles_sh[j] = Tile{0, pairs + j * cut.shared, min(cut.shared, T - j * cut.shared)};
  if (e == 0) {
    n_tiles[0] = n_wide;
    n_tiles[1] = nsh;
    n_tiles[2] = total_full + nparts - n_wide;
  }
}

// Places in expert order, stable in the pair index. A thread per pair: pairs of one warp with the same
// expert are told apart by their lanes, the warps' counts by a prefix over the block's 16 warps, so
// that nothing is serial but that prefix (one warp walking the 512 pairs took 24 us at any T).
__global__ void __launch_bounds__(kChunk)
k_route_place(const int32_t* __restrict__ ids, const float* __restrict__ w, int stride, int pairs,
              int k, int E, const int32_t* __restrict__ blockcnt, const int32_t* __restrict__ eoff,
              int32_t* __restrict__ tokidx, float* __restrict__ pw, int32_t* __restrict__ pairids) {
  __shared__ __align__(4) uint16_t before[kChunk / 32][kMaxExperts];  // pairs of an expert: per warp, then in the warps before
  __shared__ int start[kMaxExperts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_trigger();
  for (int i = threadIdx.x; i < (int)sizeof(before) / 4; i += kChunk) ((uint32_t*)before)[i] = 0;
  pdl_wait();
  const int p = blockIdx.x * kChunk + threadIdx.x;
  const bool live = p < pairs;
  const int t = live ? p / k : 0, s = live ? p % k : 0;
  const int e = live ? ids[(size_t)t * stride + s] : -1;
  const bool good = (unsigned)e < (unsigned)E;
  const float wt = live ? w[(size_t)t * stride + s] : 0.f;
  for (int i = threadIdx.x; i < E; i += kChunk) start[i] = eoff[i] + blockcnt[(size_t)blockIdx.x * E + i];
  __syncthreads();
  const unsigned same = __match_any_sync(0xffffffffu, good ? e : -1);
  if (good && lane == __ffs(same) - 1) before[warp][e] = (uint16_t)__popc(same);
  __syncthreads();
  for (int i = threadIdx.x; i < E; i += kChunk) {
    int run = 0;
#pragma unroll
    for (int v = 0; v < kChunk / 32; v++) {
      const int n = before[v][i];
      before[v][i] = (uint16_t)run;
      run += n;
    }
  }
  __syncthreads();
  if (!live) return;
  const int row = good ? start[e] + before[warp][e] + __popc(same & ((1u << lane) - 1u)) : -1;
  if (good) {
    tokidx[row] = t;
    pw[row] = wt;
  }
  // slot in the token's reduce order: ascending expert id; equal ids keep their slot order,
  // so every slot is written; a dropped pair's slot holds -1 (the combine skips it)
  int rank = 0;
  const int key = good ? e : kBadKey;
  for (int q = 0; q < k; q++) {
    const int eq = ids[(size_t)t * stride + q];
    const int kq = (unsigned)eq < (unsigned)E ? eq : kBadKey;  // dropped pairs sort behind every expert
    rank += (kq < key) || (kq == key && q < s);
  }
  pairids[(size_t)t * k + rank] = row;
}

// Scalar sigmoid gate of the shared expert (src/ref.cpp:623-626, 635): one warp per token.
// Also appends the shared expert's rows (token order) behind the routed rows.
__global__ void __launch_bounds__(256)
k_shared_gate(const uint16_t* __restrict__ x, const uint16_t* __restrict__ gw, int T, int d, int k,
              int32_t* __restrict__ tokidx, float* __restrict__ pw, float* __restrict__ sgate) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 8 + warp;
  if (t >= T) return;
  double a = 0;
  for (int c = lane; c < d; c += 32)
    a += (double)bf16_bits_to_f32(gw[c]) * (double)bf16_bits_to_f32(x[(size_t)t * d + c]);
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    int lo = __shfl_xor_sync(0xffffffffu, __double2loint(a), o);
    int hi = __shfl_xor_sync(0xffffffffu, __double2hiint(a), o);
    a += __hiloint2double(hi, lo);
  }
  if (lane == 0) {
    float g = sigmoid_f32((float)a);
    sgate[t] = g;
    tokidx[(size_t)T * k + t] = t;
    pw[(size_t)T * k + t] = g;
  }
}

}  // namespace

cudaError_t launch_router_topk(const float* logits, int T, int E, int k, int32_t* ids, float* w,
                               int stride, cudaStream_t st) {
  return launch_pdl(k_router_topk, dim3((T + kRouterWarps - 1) / kRouterWarps), dim3(kRouterWarps * 32), 0, st, logits, T, E,
                    k, ids, w, stride);
}

bool route_block_supported(int T, int k) { return T <= 16 && T * k <= kSmallPairs; }

cudaError_t launch_route_block(const RouteIn& q, cudaStream_t st) {
  static_assert(kRouteBlockBytes <= 48 * 1024, "opt-in size");
  return launch_pdl(k_route_block, dim3(1), dim3(1024), (size_t)kRouteBlockBytes, st, q);
}

cudaError_t launch_route(const RouteBuffers& rb, const int32_t* ids, const float* w, int stride,
                         int T, int k, int E, const TileCut& cut, cudaStream_t st, int* launches) {
  const int pairs = T * k;
  const int nblk = (pairs + kChunk - 1) / kChunk;
  // Every kernel of the chain waits for the one before it: its launch and set-up overlap that one's tail.
  // (These kernels with a thread per pair: 592 -> 559 us on a 77-token call, 531 -> 500 on 500 tokens.)
  cudaError_t e = launch_pdl(k_route_count, dim3(nblk), dim3(kChunk), 0, st, ids, stride, pairs, k, E, rb.blockcnt, rb.status);
  if (e == cudaSuccess)
    e = launch_pdl(k_route_scan, dim3(1), dim3(kMaxExperts), 0, st, rb.blockcnt, nblk, E, pairs, T, cut, rb.eoff, rb.runs,
                   rb.n_runs, rb.tiles, rb.tiles_narrow, rb.tiles_sh, rb.n_tiles, rb.tiles_dense, rb.dense_experts, rb.n_dense);
  if (e == cudaSuccess)
    e = launch_pdl(k_route_place, dim3(nblk), dim3(kChunk), 0, st, ids, w, stride, pairs, k, E, rb.blockcnt, rb.eoff, rb.tokidx,
                   rb.pw, rb.pairids);
  if (launches) *launches += 3;
  return e;
}

cudaError_t launch_shared_gate(const void* x_bf16, const uint16_t* gate_w_bf16, int T, int d, int k,
                               const RouteBuffers& rb, cudaStream_t st) {
  k_shared_gate<<<(T + 7) / 8, 256, 0, st>>>((const uint16_t*)x_bf16, gate_w_bf16, T, d, k,
                                             rb.tokidx, rb.pw, rb.sgate);
  return cudaGetLastError();
}

// ---- expert parallelism ---------------------------------------------------------------
// ids <- place[ids]: experts renumbered so that rank r owns the ids [r*E/G, (r+1)*E/G).
__global__ void k_apply_placement(int32_t* __restrict__ ids, int stride, int T, int k, int E,
                                  const int32_t* __restrict__ place) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < T * k) {
    int32_t* q = ids + (size_t)(p / k) * stride + p % k;
    if ((unsigned)*q < (unsigned)E) *q = place[*q];
  }
}

// Work list of the receiving rank. The receive buffer holds, source rank after source rank,
// that source's rows for this rank's experts in ascending expert order; eoff_all[s] is source
// s's expert offset table (E+1 entries). One thread per (source, local expert) segment:
// its position in the buffer, then tiles of at most tile_cap rows (full tiles first, ragged
// ones by descending size), exactly as the single-GPU tile list is built.
//
// part 4 (the other ranks' rows with their TAILS MERGED by expert): the receive buffer is
// source-major, so an expert that got rows from seven ranks has seven segments there and up to
// seven ragged tiles. Full tiles of a segment stay where they are; the rows behind a segment's
// last full tile (its tail) are copied behind the received rows, expert after expert, and tiled
// there: one ragged tile per expert instead of one per (source, expert). segs[] lists the tails in
// the order of their destination, {first row in the receive buffer, first row in the merged area,
// rows}; counts[1] = received rows R (the merged area starts there), counts[2] = merged rows (0
// when the buffer has no room for them behind R: the list is then part 2's).
__global__ void __launch_bounds__(kMaxExperts)
k_ep_tiles(const int32_t* __restrict__ eoff_all, int G, int E, int e0, int El, int tile_cap, int own, int part,
           Tile* __restrict__ tiles, int32_t* __restrict__ n_tiles, int32_t* __restrict__ counts,
           int32_t* __restrict__ segs, int cap_rows) {
  __shared__ int s_a[kMaxExperts], s_c[kMaxExperts];
  const int tid = threadIdx.x;
  const int src = tid / El, e = tid % El;
  const bool live = tid < G * El;
  int cnt = 0, first = 0;
  if (live) {
    const int32_t* eo = eoff_all + (size_t)src * (E + 1);
    cnt = eo[e0 + e + 1] - eo[e0 + e];
    first = eo[e0 + e] - eo[e0];                      // offset inside the source's segment
    for (int s2 = 0; s2 < src; s2++) {                // segments of the sources before it
      const int32_t* e2 = eoff_all + (size_t)s2 * (E + 1);
      first += e2[e0 + El] - e2[e0];
    }
    // part 1: only the rows this rank sent to itself; part 2 and 4: only the other ranks' rows;
    // part 3: this rank's own rows where they lie in its SEND buffer (row = its own expert offset)
    if ((part == 1 && src != own) || ((part == 2 || part == 4) && src == own) || (part == 3 && src != own)) cnt = 0;
    if (part == 3) first = eo[e0 + e];
  }
  int R = 0;  // rows of the source-major layout
  for (int s2 = 0; s2 < G; s2++) {
    const int32_t* e2 = eoff_all + (size_t)s2 * (E + 1);
    R += e2[e0 + El] - e2[e0];
  }
  // tiles of this thread: nf_a full tiles from first, nf_b full tiles from first_b, one ragged tile
  int nf_a = cnt / tile_cap, nf_b = 0, first_b = 0, rag = cnt % tile_cap, rag_first = first + nf_a * tile_cap;
  int merged_rows = 0;
  if (part == 4) {
    const int tail = rag;
    s_c[tid] = tail;
    __syncthreads();
    int before = 0, ttot = 0;  // tail rows of expert e from the sources before this one, from all
    if (live)
      for (int s2 = 0; s2 < G; s2++) {
        const int c2 = s_c[s2 * El + e];
        ttot += c2;
        before += s2 < src ? c2 : 0;
      }
    __syncthreads();
    if (tid < El) s_a[tid] = ttot;
    __syncthreads();
    int tbase = 0, all_tails = 0;  // tail rows of the experts before e, of all experts
    for (int e2 = 0; e2 < El; e2++) {
      all_tails += s_a[e2];
      tbase += e2 < e ? s_a[e2] : 0;
    }
    __syncthreads();
    if (R + all_tails <= cap_rows) {
      merged_rows = all_tails;
      if (live) {
        int32_t* sg = segs + 3 * (e * G + src);   // destination order: expert-major
        sg[0] = rag_first;
        sg[1] = R + tbase + before;
        sg[2] = tail;
      }
      // the tail leaves this thread; the thread of source 0 tiles the expert's merged tails
      rag = 0;
      if (live && src == 0) {
        nf_b = ttot / tile_cap;
        first_b = R + tbase;
        rag = ttot % tile_cap;
        rag_first = first_b + nf_b * tile_cap;
      }
    }
  }
  const int nfull = nf_a + nf_b;
  s_c[tid] = nfull;
  __syncthreads();
  for (int o = 1; o < kMaxExperts; o <<= 1) {
    const int c = tid >= o ? s_c[tid - o] : 0;
    __syncthreads();
    s_c[tid] += c;
    __syncthreads();
  }
  const int total_full = s_c[kMaxExperts - 1], full0 = s_c[tid] - nfull;
  for (int j = 0; j < nf_a; j++) tiles[full0 + j] = Tile{e, first + j * tile_cap, tile_cap};
  for (int j = 0; j < nf_b; j++) tiles[full0 + nf_a + j] = Tile{e, first_b + j * tile_cap, tile_cap};
  s_a[tid] = rag;
  __syncthreads();
  int rank = 0, nparts = 0;
  for (int o = 0; o < kMaxExperts; o++) {
    const int pp = s_a[o];
    nparts += pp > 0;
    rank += (pp > rag) || (pp == rag && o < tid);
  }
  if (rag > 0) tiles[total_full + rank] = Tile{e, rag_first, rag};
  if (tid == 0) {
    n_tiles[0] = total_full + nparts;
    counts[0] = R;
    counts[1] = merged_rows;
  }
}

cudaError_t launch_apply_placement(int32_t* ids, int stride, int T, int k, int E, const int32_t* place,
                                   cudaStream_t st) {
  k_apply_placement<<<(T * k + 255) / 256, 256, 0, st>>>(ids, stride, T, k, E, place);
  return cudaGetLastError();
}

cudaError_t launch_ep_tiles(const int32_t* eoff_all, int G, int E, int e0, int El, int tile_cap,
                            Tile* tiles, int32_t* n_tiles, int32_t* counts, cudaStream_t st, int own, int part,
                            int32_t* segs, int cap_rows) {
  if (part == 4 && !segs) return cudaErrorInvalidValue;
  k_ep_tiles<<<1, kMaxExperts, 0, st>>>(eoff_all, G, E, e0, El, tile_cap, own, part, tiles, n_tiles, counts, segs, cap_rows);
  return cudaGetLastError();
}

// The tails of part 4 copied into the merged area behind the received rows: one warp per merged
// row; its segment is found by bisection in segs[] (in destination order; empty segments share
// their first row with the next one, so the LAST segment starting at or before the row holds it).
// rowmap[merged row - R] = the row's place in the source-major layout: the down GEMM writes the
// result there, so that results leave in the senders' order without another pass.
__global__ void __launch_bounds__(256)
k_ep_merge_tails(uint4* __restrict__ x_recv, const int32_t* __restrict__ segs, int n_seg,
                 const int32_t* __restrict__ counts, int per_row, int32_t* __restrict__ rowmap) {
  __shared__ int s_src[kMaxExperts], s_dst[kMaxExperts];
  for (int i = threadIdx.x; i < n_seg; i += blockDim.x) {
    s_src[i] = segs[3 * i];
    s_dst[i] = segs[3 * i + 1];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int R = counts[0], rows = counts[1];
  const int n_warps = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < rows; i += n_warps) {
    const int dst = R + i;
    int lo = 0, hi = n_seg - 1;
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (s_dst[m] <= dst) lo = m; else hi = m - 1;
    }
    const int j = s_src[lo] + (dst - s_dst[lo]);
    const uint4* src = x_recv + (size_t)j * per_row;
    uint4* out = x_recv + (size_t)dst * per_row;
    for (int v = lane; v < per_row; v += 32) out[v] = src[v];
    if (lane == 0) rowmap[i] = j;
  }
}

cudaError_t launch_ep_merge_tails(__half* x_recv, const int32_t* segs, int n_seg, const int32_t* counts, int d,
                                  int32_t* rowmap, int sms, cudaStream_t st) {
  k_ep_merge_tails<<<sms * 4, 256, 0, st>>>((uint4*)x_recv, segs, n_seg, counts, d / 8, rowmap);
  return cudaGetLastError();
}

// Waits until every one of n flags (written by peer GPUs' copy engines behind their data)
// has reached `expected`. Bounded: after 2 s the kernel records status {3, index of the
// missing flag} and returns, so that the context stays usable and the host sees the timeout.
__global__ void k_wait_flags(const int32_t* flags, int n, int32_t expected, int32_t* status) {
  const int i = threadIdx.x;
  if (i >= n) return;
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (uint32_t spin = 0;; spin++) {
    int32_t v;
    asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flags + i) : "memory");
    if (v - expected >= 0) return;
    if ((spin & 63u) == 63u) {
      unsigned long long t1;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      if (t1 - t0 > 2000000000ull) {
        if (atomicCAS(status, 0, 3) == 0) status[1] = i;
        return;
      }
      __nanosleep(200);
    }
  }
}

cudaError_t launch_wait_flags(const int32_t* flags, int n, int32_t expected, int32_t* status, cudaStream_t st) {
  k_wait_flags<<<1, 32, 0, st>>>(flags, n, expected, status);
  return cudaGetLastError();
}

int route_chunk() { return kChunk; }

}  // namespace b200moe
