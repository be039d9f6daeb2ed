// expert_dense.cu -- the down GEMM of popular experts in long chunks (sm_100a): their weights are expanded once per call to the
// fp16 values that the grouped dequant-GEMM (expert_tc.cu) forms for every 192 rows anew, and multiplied by a plain grouped GEMM
// on pairs of SMs (tcgen05 cta_group::2): bit for bit the same results. A group of 768 rows is four tiles there and three here.
//
// k_expand: bound by the HBM, 10.5 MB per expert of 4096 x 1024: 28 experts in 61 us = 4.8 TB/s (a row's 128 bytes written by eight lanes
// with 16-byte stores: 79 us).
// k_expert_dense: a pair of CTAs multiplies 256 tokens x 256 weight rows, each CTA holding 128 rows of both operands of a K block in
// one of six stages of 32 KB, two accumulators of 256 columns. Tokens are the M side, so that an epilogue thread has 32 contiguous
// output columns of its token and stores whole sectors without a transposition. Bound by the tensor pipe: 1473 TFLOP/s at 145k rows
// of 4096 x 1024 (0.90 of the measured burst), where the dequant-GEMM's down launch makes 1018: its tiles of 8 pairs of K blocks are too
// short to hide the handshake between decoding and MMAs. Two warps issue the copies: a thread starts one every ~170
// cycles, and a K block's MMAs take 512. Both CTAs' copies complete on the first one's barriers, so
// that no thread relays "landed" between them; what else crosses (an accumulator is free) is an arrival with .release.cluster, and all waits are
// .acquire.cluster. That costs 0.6 %: 708 us of a 16384-token call's launch against 704 with arrivals and waits of one CTA's scope and a relay. A
// relay with .release.cluster took 1800 cycles per K block, a fence.acq_rel.cluster behind the MMA warp's waits 775 each.
#include "tc_dev.cuh"

namespace b200moe {

namespace {

// ---- expansion ------------------------------------------------------------------------
constexpr int kExpandThreads = 512;

__device__ __forceinline__ void st_global_32(void* p, const uint32_t* v) {  // a whole sector
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

template <int FMT>
__global__ void __launch_bounds__(kExpandThreads)
k_expand(const Image img, const int32_t* __restrict__ experts, const int32_t* __restrict__ n_dense, __half* __restrict__ out) {
  __shared__ uint32_t pair_table[256 * 32];  // a copy per lane
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 256 * 32; i += kExpandThreads) {
    const __half2 v = __floats2half2_rn(img.book[(i >> 5) & 15], img.book[i >> 9]);
    pair_table[i] = *(const uint32_t*)&v;
  }
  pdl_trigger();
  pdl_wait();
  __syncthreads();
  const int KB = img.n_kblocks, K = KB * kTileK, n_slots = n_dense[1];
  const int rows = img.n_mtiles * kTileM;
  // a warp takes a sub-block column of 32 rows, four K blocks of it at a time; a lane decodes its row
  const int strips = (KB + 3) >> 2, per_slot = img.n_mtiles * (kTileM / kSubRows) * strips;
  constexpr int sub_b = sub_bytes(FMT);
  const uint32_t* const table = pair_table + lane;
  for (long long u = (long long)blockIdx.x * (kExpandThreads / 32) + warp; u < (long long)n_slots * per_slot;
       u += (long long)gridDim.x * (kExpandThreads / 32)) {
    const int slot = (int)(u / per_slot), v = (int)(u % per_slot);
    const int strip = v % strips, sub = (v / strips) & 3, mt = v / (strips * 4);
    const uint8_t* sb = img.mtile(experts[slot], mt) + ((size_t)sub * KB + 4 * strip) * sub_b;
    const int row = mt * kTileM + sub * kSubRows + lane;
    __half* o = out + ((size_t)slot * rows + row) * K + (size_t)strip * 4 * kTileK;
    const int nk = min(4, KB - 4 * strip);
#pragma unroll 2
    for (int kb = 0; kb < nk; kb++, sb += sub_b, o += kTileK) {
      const uint4 c[2] = {__ldg((const uint4*)(sb + lane * 16)), __ldg((const uint4*)(sb + kHalfBytes + lane * 16))};
      const uint8_t* pm = sb + kSubCodes + lane * meta_row_bytes(FMT);
      RowMetaTc sc{0, 0, 0, 0};
      if (FMT == kQ4CP) {
        sc.a = __ldg((const uint32_t*)pm);
      } else {
        const uint4 t = __ldg((const uint4*)pm);
        sc = RowMetaTc{t.x, t.y, t.z, t.w};
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        GroupDecode<FMT> gd;
        gd.init(sc, h);
        const uint32_t w4[4] = {c[h].x, c[h].y, c[h].z, c[h].w};
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
          uint32_t w[8];
#pragma unroll
          for (int b = 0; b < 8; b++) {
            const __half2 x2 = gd.weight(table[((w4[q + (b >> 2)] >> (8 * (b & 3))) & 255u) * 32], q * 4 + b);
            w[b] = *(const uint32_t*)&x2;
          }
          st_global_32(o + h * 32 + q * 8, w);
        }
      }
    }
  }
}

// ---- grouped GEMM ---------------------------------------------------------------------
constexpr int kStages = 6;
constexpr int kOperand = 128 * 128;         // bytes of 128 rows x 64 halfs
constexpr int kStageBytes = 2 * kOperand;   // 128 rows of activations, 128 of weights
constexpr int kDenseThreads = 256;          // warps 0 and 3 copies, 1 MMAs (of both CTAs, in the first), 2 tensor memory, 4-7 epilogue
constexpr int kDenseSmem = kStages * kStageBytes + 1024 + 1024;  // + alignment + barriers
constexpr int kAcc = 256;                   // columns of an accumulator

struct DenseParams {
  const Tile* tiles;         // {place among the expanded experts, first row, 256}
  const int32_t* n_dense;    // [0] tiles
  __half* out;
  int out_ld;
  int KB, n_ntiles;          // K / 64, tiles of 256 weight rows per expert
  int32_t* status;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t of_leader(uint32_t addr) {  // the same place in the pair's first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// Orders what this thread did before for the other CTA's thread that waits for it (mbar_wait<true>).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// A copy into this CTA's shared memory whose bytes are counted on a barrier of the pair's other CTA, or its own.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {  // arrives on that barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kDenseThreads, 1)
k_expert_dense(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const DenseParams p) {
  extern __shared__ uint8_t dense_raw[];
  const uint32_t raw = smem_u32(dense_raw);
  const uint32_t ring = (raw + 1023) & ~1023u, bars = ring + kStages * kStageBytes;
  uint8_t* const bar_ptr = dense_raw + (bars - raw);
  constexpr uint32_t kFull = 0, kEmpty = 8 * kStages, kAccFull = 16 * kStages, kAccEmpty = kAccFull + 16;
  volatile int* abort_flag = (volatile int*)(bar_ptr + kAccEmpty + 16);
  uint32_t* tmem_slot = (uint32_t*)(bar_ptr + kAccEmpty + 24);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  pdl_wait();
  pdl_trigger();  // (behind the wait: the launches behind this one run beside it)
  if (p.n_dense[0] == 0) return;  // (all CTAs)
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; i++) {
      mbar_init(bars + kFull + 8 * i, 2);  // the first CTA's two copying warps, with both CTAs' byte counts (the second's is not used)
      mbar_init(bars + kEmpty + 8 * i, 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(bars + kAccFull + 8 * i, 1);
      mbar_init(bars + kAccEmpty + 8 * i, 8);  // epilogue warps of both CTAs (the leader's is the one in use)
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  const int n_items = p.n_dense[0] * p.n_ntiles;
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int KB = p.KB;

  if (warp == 0 || warp == 3) {
    // ================= copies: this CTA's 128 rows of activations (warp 0) and of weights (warp 3) =================
    if (lane == 0) {
      const CUtensorMap* map = warp == 0 ? &map_x : &map_w;
      const uint32_t off = warp == 0 ? 0 : kOperand;
      uint32_t stage = 0, ph = 0;
      bool ok = true;
      for (int it = cluster; it < n_items && ok; it += n_clusters) {
        const Tile t = p.tiles[it / p.n_ntiles];
        const int row = (warp == 0 ? t.first : (t.expert * p.n_ntiles + it % p.n_ntiles) * 256) + (int)rank * 128;
        for (int kb = 0; kb < KB; kb++) {
          ok = mbar_wait<true>(bars + kEmpty + 8 * stage, ph ^ 1, abort_flag, p.status, 21);
          if (!ok) break;
          // (the second CTA's bytes may come in before the first has announced them: the phase ends with its arrivals at the earliest, and
          // is the same, since a stage is free only when the MMAs that waited for the phase before are done)
          const uint32_t bar = bars + kFull + 8 * stage;
          if (rank == 0) mbar_expect_tx(bar, 2 * kOperand);
          tma_load_2d_pair(ring + stage * kStageBytes + off, map, kb * kTileK, row, of_leader(bar));
          if (++stage == (uint32_t)kStages) {
            stage = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ================= MMA issue, for both CTAs =================
    const uint32_t idesc = (1u << 4) | (256u / 8 << 17) | (256u / 16 << 24);  // D fp32, A and B fp16, both K-major
    uint32_t stage = 0, ph = 0, li = 0;
    bool ok = true;
    for (int it = cluster; it < n_items && ok; it += n_clusters, li++) {
      const uint32_t acc = li & 1, accph = (li >> 1) & 1;
      ok = __all_sync(0xffffffffu, mbar_wait<true>(bars + kAccEmpty + 8 * acc, accph ^ 1, abort_flag, p.status, 23));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem + acc * kAcc;
      for (int kb = 0; kb < KB; kb++) {
        ok = __all_sync(0xffffffffu, mbar_wait<true>(bars + kFull + 8 * stage, ph, abort_flag, p.status, 24));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t a = b_descriptor(ring + stage * kStageBytes), b = b_descriptor(ring + stage * kStageBytes + kOperand);
#pragma unroll
          for (int ks = 0; ks < 4; ks++) mma_pair(d_tmem, a + ks * 2, b + ks * 2, idesc, (kb | ks) != 0 ? 1u : 0u);
          commit_pair(bars + kEmpty + 8 * stage);
          if (kb == KB - 1) commit_pair(bars + kAccFull + 8 * acc);
        }
        __syncwarp();
        if (++stage == (uint32_t)kStages) {
          stage = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp >= 4) {
    // ================= epilogue: a thread has a token's row =================
    const int quarter = warp & 3;
    uint32_t li = 0;
    for (int it = cluster; it < n_items; it += n_clusters, li++) {
      const Tile t = p.tiles[it / p.n_ntiles];
      const int nt = it % p.n_ntiles;
      const uint32_t acc = li & 1, accph = (li >> 1) & 1;
      if (!__all_sync(0xffffffffu, mbar_wait<true>(bars + kAccFull + 8 * acc, accph, abort_flag, p.status, 25))) break;
      tc_fence_after();
      const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + acc * kAcc;
      const int r = (int)rank * 128 + quarter * 32 + lane;
      __half* const orow = p.out + (size_t)(t.first + r) * p.out_ld + nt * 256;
      for (int c0 = 0; c0 < 256; c0 += 32) {
        uint32_t v[32], o[16];
        tc_ld32(src + c0, v);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; j += 2)  // finite values saturate to the fp16 range, NaN stays NaN
          asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(o[j / 2]) : "f"(__uint_as_float(v[j + 1])), "f"(__uint_as_float(v[j])));
        if (r < t.count) {
          st_global_32(orow + c0, o);
          st_global_32(orow + c0 + 16, o + 8);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(of_leader(bars + kAccEmpty + 8 * acc));
    }
  }

  // ---- teardown: neither CTA leaves while the other may still read its memory or arrive on its barriers ----
  __syncthreads();
  if (*abort_flag) {
    const unsigned long long t0 = now_ns();
    while (now_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  cluster_sync();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int FMT>
cudaError_t expand(const TcPlan* plan, const Image& img, const int32_t* experts, const int32_t* n_dense, __half* out, cudaStream_t st) {
  return launch_pdl(k_expand<FMT>, dim3(plan->sms * 3), dim3(kExpandThreads), 0, st, img, experts, n_dense, out);
}

}  // namespace

cudaError_t launch_expand(const TcPlan* plan, const Image& img, const int32_t* experts, const int32_t* n_dense, __half* out,
                          cudaStream_t st) {
  if (img.act_shift || img.paired || plan->margin > 0) return cudaErrorNotSupported;
  if (img.fmt == kQ51) return expand<kQ51>(plan, img, experts, n_dense, out, st);
  if (img.fmt != kQ4CP) return cudaErrorNotSupported;
  return expand<kQ4CP>(plan, img, experts, n_dense, out, st);
}

cudaError_t launch_down_dense(const TcPlan* plan, const Tile* tiles, const int32_t* n_dense, int d, int mid, __half* pairs16, int32_t* status,
                              cudaStream_t st) {
  if (plan->margin > 0) return cudaErrorNotSupported;  // its pairs fill the GPU and start early: not beside exchange kernels
  static OncePerDevice once;
  if (cudaError_t e = once([] { return cudaFuncSetAttribute(k_expert_dense, cudaFuncAttributeMaxDynamicSharedMemorySize, kDenseSmem); })) return e;
  const DenseParams p{tiles, n_dense, pairs16, d, mid / kTileK, d / 256, status};
  return launch_pdl(k_expert_dense, dim3(plan->sms / 2 * 2), dim3(kDenseThreads), (size_t)kDenseSmem, st, plan->h[2], plan->w_dense, p);
}

}  // namespace b200moe
