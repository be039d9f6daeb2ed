// expert_few.cu -- grouped dequant-GEMM for tiles of at most 64 rows (tcgen05, sm_100a): expert_tc.cu's operands and results,
// bit for bit, for experts with few rows, whose MMAs are so short that the decoding of the weights decides.
//
// One CTA per SM, 24 warps, K blocks (64 wide) in quads:
//   warp 0      producer of activations: one tensor copy per pair of K blocks (boxes of 16, 32, 48 or 64 rows), counted by the
//               barrier that the quad's dequantising warps arrive on
//   warp 1      sixteen tcgen05.mma per quad behind ONE barrier check, which is made (without blocking) behind the quad before
//   warp 2      producer of packed weights: four bulk copies per quad into a ring of 4 stages (3 in the Q5_1 form)
//   warps 4-19  dequantise, two sets of eight that alternate quads; a thread decodes its weight row of two K blocks of a quad, 32
//               codes at a time (a table lookup per code byte, see Map in expert_tc.cu), into tensor memory. The stores are
//               waited for behind the next quad's first 32 codes.
//   warps 20-23 epilogue, 16 rows of the expert at a time; two accumulators, three slots of 128 columns for the weights
// What bounds it: of a 128 x 64 block's 255 cycles (12 rows; 512 experts of 4096 x 1024, 600 tokens, 505 us of the gate/up
// launch at 4.8 TB/s) the table lookups take 126 by themselves, the stores to tensor memory another 90 (they and the loads share
// a pipe), the MMAs' reads of it the rest; weights from L2 instead of HBM gain 2 %, no epilogue 1 %. The HBM's share is 200. Before,
// with pairs of K blocks as the unit, a relay warp and two more barrier checks of the MMA warp (each ~180 cycles of its
// serial chain): 375 cycles, 650 us. Steps: quads alone 714 us; activations counted by the weights' barrier, checks ahead of their
// use, third slot, stores waited for later 519; stores of 16 columns instead of 32 503.
#include "tc_dev.cuh"

namespace b200moe {

namespace {

constexpr int kRows = kTcNarrowN;
constexpr int kNS = 3;                 // tensor-memory A slots; a slot holds a quad of K blocks (128 columns)
constexpr int kThreads = 768;          // 24 warps: 4 service, 16 dequantising, 4 epilogue
constexpr int kTmemA = 2 * kRows;      // first column of the A slots, behind two accumulators
static_assert(kTmemA + kNS * 128 <= 512, "tensor memory: two accumulators and the A slots");

// Shared memory in absolute addresses (see Map in expert_tc.cu: the pair table on a 64 KB boundary).
constexpr int kOffBar = 2048, kOffU = 3072, kOffX = 11264, kOffLut = 65536, kOffW = 131072, kSmemEnd = 233472;
constexpr int kSmemBytes = kSmemEnd - 1024;  // dynamic bytes requested: the allocation starts at 1 KB
// Activations of a pair of K blocks: 4, 8, 12 or 16 KB by the rows of the tile's box (16, 32, 48, 64). Two quads of 48 or 64 rows
// or three of fewer fit below the table, but for the last pair of 64 rows, which lies behind it.
constexpr int kPair64 = kRows * 256, kOffX3 = kOffLut + 65536, kOffStages = kOffX3 + kPair64;
static_assert(kOffX + 3 * kPair64 <= kOffLut && kOffX3 == kOffW, "activations");
constexpr uint32_t stage_bytes(int fmt) { return 16 * (uint32_t)sub_bytes(fmt); }        // four sub-blocks x four K blocks
constexpr int stages(int fmt) { return (kSmemEnd - kOffStages) / (int)stage_bytes(fmt); }  // 4, 4, 3
constexpr int kMaxStages = 4;

constexpr int kBarAFull = 0,                      // [A slot] a quad's weights are in tensor memory, its activations have landed
              kBarADone = kBarAFull + kNS,        // [A slot] all its MMAs have completed
              kBarAccFull = kBarADone + kNS,
              kBarAccEmpty = kBarAccFull + 2,
              kBarCFull = kBarAccEmpty + 2,       // [weight stage] a quad's packed tiles have landed
              kBarCEmpty = kBarCFull + kMaxStages,
              kNumBars = kBarCEmpty + kMaxStages;
static_assert(kNumBars * 8 + 16 + 32 <= 1024, "barrier block too small");

// Where a quad's activations lie. Slots of another size than the last tile's start afresh (tiles come by size, so that this
// is rare); their producer then waits for all MMAs before.
struct XSlots {
  uint32_t rows = 0, n = 0, i = 0;  // rows of the box, slots of that size, the next quad's
  __device__ __forceinline__ static uint32_t box(int count) { return (count + 15) & ~15; }
  __device__ __forceinline__ bool resize(int count) {  // true: the size is another one
    if (rows == box(count)) return false;
    rows = box(count);
    n = rows > 32 ? 2 : 3;
    i = 0;
    return true;
  }
  __device__ __forceinline__ uint32_t addr(int h) const {
    const uint32_t pair = 2 * i + h;
    return rows == 64 && pair == 3 ? (uint32_t)kOffX3 : (uint32_t)kOffX + pair * rows * 256;
  }
  __device__ __forceinline__ void next() {
    if (++i == n) i = 0;
  }
};

// A look at a barrier that does not block: its answer is used some work later.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

struct FewParams {
  Image img;
  const Tile* tiles;
  const int32_t* n_tiles;
  __half* out;
  int out_ld;  // mid (gate/up) or d (down)
  int32_t* status;
  int beside;      // 1: runs beside the launch in front of it (see the wait in the set-up)
  int early_next;  // 1: the next launch of the stream may start its set-up while this one runs
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(0), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

template <bool UP, bool DUAL, int FMT>
__global__ void __launch_bounds__(kThreads, 1)
k_expert_few(const __grid_constant__ CUtensorMap map16, const __grid_constant__ CUtensorMap map32,
             const __grid_constant__ CUtensorMap map48, const __grid_constant__ CUtensorMap map64, const FewParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t dyn0 = smem_u32(smem_raw);
  uint8_t* const smem = smem_raw - dyn0;  // smem + A is the generic pointer of absolute shared address A
  {
    uint32_t dyn_size;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
    if (dyn0 > (uint32_t)kOffBar || dyn0 + dyn_size < (uint32_t)kSmemEnd) {
      // the fixed map does not fit this launch: refuse (uniform for the whole CTA)
      if (threadIdx.x == 0 && atomicCAS(p.status, 0, 2) == 0) p.status[1] = (int)dyn0;
      return;
    }
  }
  constexpr uint32_t bars = kOffBar;
  constexpr int kNST = stages(FMT);
  static_assert(kNST <= kMaxStages, "barrier block");
  volatile int* abort_flag = (volatile int*)(smem + kOffBar + kNumBars * 8);
  uint32_t* tmem_slot = (uint32_t*)(smem + kOffBar + kNumBars * 8 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (a launch beside another one starts only when its list is there, see below: with none, it just keeps the order)
  if (p.beside && p.n_tiles[0] == 0) {
    pdl_trigger();
    if (blockIdx.x == 0) pdl_wait();
    return;
  }
  const Image img = p.img;
  const int KB = img.n_kblocks;

  // ---- set-up (weights and the CTA's own state only: it overlaps the tail of the kernel before) ----
  if (threadIdx.x == 0) {
    for (int i = 0; i < kNS; i++) {
      mbar_init(bars + 8 * (kBarAFull + i), 9);  // the set's dequantising warps, the activations' producer (with byte count)
      mbar_init(bars + 8 * (kBarADone + i), 1);
    }
    for (int i = 0; i < kNST; i++) {
      mbar_init(bars + 8 * (kBarCFull + i), 1);
      mbar_init(bars + 8 * (kBarCEmpty + i), 8);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(bars + 8 * (kBarAccFull + i), 1);
      mbar_init(bars + 8 * (kBarAccEmpty + i), 4);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  // pair table: entry b = (f16(book[b & 15]), f16(book[b >> 4])), one private copy per lane
  for (int i = threadIdx.x; i < (DUAL ? 2 : 1) * 256 * 32; i += kThreads) {
    const int half_id = i >> 13, entry = (i >> 5) & 255;
    const float lo = img.book[half_id * 16 + (entry & 15)], hi = img.book[half_id * 16 + (entry >> 4)];
    *(__half2*)(smem + kOffLut + entry * 256 + half_id * 128 + (i & 31) * 4) = __floats2half2_rn(lo, hi);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // (wait and trigger: as in k_expert_tc)
  if (!p.beside) pdl_wait();
  if (p.early_next) pdl_trigger();
  const int n_items = p.n_tiles[0] * img.n_mtiles;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  const int NP = (KB + 1) >> 1, NQ = (KB + 3) >> 2;  // pairs and quads of K blocks of an item
  if (warp == 0) {
    // ================= producer of activations: one tensor copy per pair of K blocks =================
    if (lane == 0) {
      XSlots xs;
      uint32_t qi = 0;
      bool ok = true;
      auto done = [&](uint32_t q) { return mbar_wait(bars + 8 * (kBarADone + q % kNS), (q / kNS) & 1, abort_flag, p.status, 2, 64); };
      Tile t_ahead = (int)blockIdx.x < n_items ? p.tiles[blockIdx.x / img.n_mtiles] : Tile{0, 0, 0};
      for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
        const Tile t = t_ahead;  // read one item ahead: its latency is off this loop's critical path
        if (it + (int)gridDim.x < n_items) t_ahead = p.tiles[(it + gridDim.x) / img.n_mtiles];
        const CUtensorMap* map = t.count <= 16 ? &map16 : t.count <= 32 ? &map32 : t.count <= 48 ? &map48 : &map64;
        if (xs.resize(t.count) && qi > 0) ok = done(qi - 1);
        for (int qq = 0; qq < NQ && ok; qq++, qi++) {
          // (the slot's last user is done, and so is the A slot's, whose barrier takes this quad's phase then)
          if (qi >= xs.n) ok = done(qi - xs.n);
          if (!ok) break;
          const int np = min(2, NP - 2 * qq);
          const uint32_t bar = bars + 8 * (kBarAFull + qi % kNS);
          mbar_expect_tx(bar, np * xs.rows * 256);  // (a K block behind the last one is filled with zeros, and counts)
          for (int h = 0; h < np; h++) tma_load_3d(xs.addr(h), map, t.first, (4 * qq + 2 * h) >> img.act_shift, bar);
          xs.next();
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issue (the whole warp runs the loop, one elected lane issues) =================
    uint32_t li = 0, aslot = 0, aph = 0;
    XSlots xs;
    bool ok = true, ready = false;  // ready: the next quad's barrier has been seen complete
    Tile t_ahead = (int)blockIdx.x < n_items ? p.tiles[blockIdx.x / img.n_mtiles] : Tile{0, 0, 0};
    for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, li++) {
      const Tile t = t_ahead;
      if (it + (int)gridDim.x < n_items) t_ahead = p.tiles[(it + gridDim.x) / img.n_mtiles];
      const uint32_t idesc = instr_desc((t.count + 15) & ~15);
      const uint32_t acc = li & 1, accph = (li >> 1) & 1;
      xs.resize(t.count);
      const uint32_t blk = img.act_shift ? 0 : xs.rows * 128 >> 4;  // from the first K block of a pair to the second
      ok = __all_sync(0xffffffffu, mbar_wait(bars + 8 * (kBarAccEmpty + acc), accph ^ 1, abort_flag, p.status, 3));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem + acc * kRows;
      for (int qq = 0; qq < NQ; qq++) {
        if (!ready) {
          ok = __all_sync(0xffffffffu, mbar_wait(bars + 8 * (kBarAFull + aslot), aph, abort_flag, p.status, 4));
          if (!ok) break;
        }
        tc_fence_after();
        const uint32_t a_tmem = tmem + kTmemA + aslot * 128, done = bars + 8 * (kBarADone + aslot);
        const int nk = KB - 4 * qq;
        if (elect_one()) {
          const uint64_t b0 = b_descriptor(xs.addr(0));
#pragma unroll
          for (int ks = 0; ks < 4; ks++) tc_mma_ts(d_tmem, a_tmem + ks * 8, b0 + (uint64_t)(ks * 2), idesc, (qq | ks) != 0 ? 1u : 0u);
          if (nk > 1) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) tc_mma_ts(d_tmem, a_tmem + 32 + ks * 8, b0 + (uint64_t)(blk + ks * 2), idesc, 1u);
          }
          if (nk > 2) {
            const uint64_t b2 = b_descriptor(xs.addr(1));
#pragma unroll
            for (int ks = 0; ks < 4; ks++) tc_mma_ts(d_tmem, a_tmem + 64 + ks * 8, b2 + (uint64_t)(ks * 2), idesc, 1u);
            if (nk > 3) {
#pragma unroll
              for (int ks = 0; ks < 4; ks++) tc_mma_ts(d_tmem, a_tmem + 96 + ks * 8, b2 + (uint64_t)(blk + ks * 2), idesc, 1u);
            }
          }
          tc_commit(done);
          if (qq == NQ - 1) tc_commit(bars + 8 * (kBarAccFull + acc));
        }
        __syncwarp();
        xs.next();
        if (++aslot == (uint32_t)kNS) {
          aslot = 0;
          aph ^= 1;
        }
        ready = __all_sync(0xffffffffu, mbar_test(bars + 8 * (kBarAFull + aslot), aph));
      }
    }
  } else if (warp == 2) {
    // ================= producer of packed weights: a bulk copy per sub-block and quad of K blocks =================
    if (lane == 0) {
      constexpr uint32_t sub_b = sub_bytes(FMT);
      const size_t col_b = (size_t)KB * sub_b;  // from one sub-block to the next
      uint32_t stage = 0, ph = 0;
      bool ok = true;
      Tile t_ahead = (int)blockIdx.x < n_items ? p.tiles[blockIdx.x / img.n_mtiles] : Tile{0, 0, 0};
      for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
        const uint8_t* src = img.mtile(t_ahead.expert, it % img.n_mtiles);
        if (it + (int)gridDim.x < n_items) t_ahead = p.tiles[(it + gridDim.x) / img.n_mtiles];
        for (int qq = 0; qq < NQ; qq++, src += 4 * sub_b) {
          ok = mbar_wait(bars + 8 * (kBarCEmpty + stage), ph ^ 1, abort_flag, p.status, 12, 64);
          if (!ok) break;
          const uint32_t bytes = (uint32_t)min(4, KB - 4 * qq) * sub_b, bar = bars + 8 * (kBarCFull + stage);
          mbar_expect_tx(bar, kTileM / kSubRows * bytes);
#pragma unroll
          for (int s = 0; s < kTileM / kSubRows; s++)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             (uint32_t)kOffStages + stage * stage_bytes(FMT) + s * (4 * sub_b)), "l"(src + s * col_b), "r"(bytes), "r"(bar)
                         : "memory");
          if (++stage == (uint32_t)kNST) {
            stage = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp >= 4 && warp < 20) {
    // ================= dequantise into tensor memory =================
    // Two sets of eight warps alternate quads; in a set, four warps (one per 32-lane quarter of tensor memory) take
    // the K blocks 0 and 2 of a quad, four 1 and 3. A thread decodes its weight row of a K block into 32 columns.
    const int set = (warp - 4) >> 3, kblk = ((warp - 4) >> 2) & 1, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lut = (uint32_t)kOffLut | (uint32_t)(DUAL && r >= 64 ? 128 : 0) | (uint32_t)(lane * 4);
    const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const uint32_t total = (uint32_t)my_items * (uint32_t)NQ;
    constexpr uint32_t sub_b = sub_bytes(FMT);
    const int pos = tile_pos(r, img.paired);
    const uint32_t row = (uint32_t)kOffStages + (uint32_t)(pos >> 5) * (4 * sub_b) + (uint32_t)kblk * sub_b + (uint32_t)code_offset(pos);
    const uint32_t off_m = (uint32_t)meta_offset(FMT, pos) - (uint32_t)code_offset(pos);
    const uint32_t a_col = tmem + ((uint32_t)(quarter * 32) << 16) + kTmemA + kblk * 32;
    struct Codes {
      uint4 half[2];
      RowMetaTc sc;
    };
    auto read = [&](uint32_t pc, Codes& c) {
      c.half[0] = lds128(pc);
      c.half[1] = lds128(pc + kHalfBytes);
      if (FMT == kQ4CP) {
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(c.sc.a) : "r"(pc + off_m));
      } else if (FMT == kQ4K) {
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(c.sc.a), "=r"(c.sc.b) : "r"(pc + off_m));
      } else {
        const uint4 u = lds128(pc + off_m);
        c.sc = RowMetaTc{u.x, u.y, u.z, u.w};
      }
    };
    // half a K block of the row: 32 codes into 16 columns
    auto decode = [&](const Codes& c, const int h, uint32_t* v) {
      GroupDecode<FMT> gd;
      gd.init(c.sc, h);
      const uint32_t w4[4] = {c.half[h].x, c.half[h].y, c.half[h].z, c.half[h].w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const uint32_t addr = __byte_perm(w4[q], lut, 0x7604u | (uint32_t)(b << 4));
          uint32_t pair;
          asm("ld.shared.b32 %0, [%1];" : "=r"(pair) : "r"(addr));
          __half2 w2 = gd.weight(pair, q * 4 + b);
          v[q * 4 + b] = *(uint32_t*)&w2;
        }
      }
    };
    uint32_t stage = (uint32_t)set, ph = 0;                    // qi % kNST, (qi / kNST) & 1
    uint32_t aslot = (uint32_t)set, aph = 1;                   // qi % kNS, parity of the phase before that use
    int qq = set % NQ;
    uint32_t pending = 0;  // the barrier of the quad whose stores are under way: they are waited for behind the next decode
    auto signal = [&]() {
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pending);
      pending = 0;  // (a wait below that gives up leaves the loop: no second arrival behind it)
    };
    // A parity wait for a stage is good only when the use before it has completed. With an even number of stages that was
    // this set's own; with an odd one the other set's quad qi - 3, whose MMAs this set then waits for first.
    constexpr bool kOdd = kNST % 2 != 0;
    static_assert(!kOdd || kNST == kNS, "the stage's and the slot's last user are the same quad");
    auto slot_free = [&]() { return (bool)__all_sync(0xffffffffu, mbar_wait(bars + 8 * (kBarADone + aslot), aph, abort_flag, p.status, 7)); };
    bool c_ready = false;
    for (uint32_t qi = (uint32_t)set; qi < total; qi += 2) {
      if (kOdd) {
        if (pending) signal();
        if (!slot_free()) break;
      }
      if (!c_ready && !__all_sync(0xffffffffu, mbar_wait(bars + 8 * (kBarCFull + stage), ph, abort_flag, p.status, 11))) break;
      const uint32_t pc = row + stage * stage_bytes(FMT);
      const int left = KB - 4 * qq - kblk;  // K blocks of the item from this thread's first one on
      const bool one = left > 0, two = left > 2;
      Codes c0 = Codes{}, c1 = Codes{};
      uint32_t va[16], vb[16];
      if (one) read(pc, c0);
      if (two) read(pc + 2 * sub_b, c1);
      const bool a_test = kOdd || mbar_test(bars + 8 * (kBarADone + aslot), aph);
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (kBarCEmpty + stage));
      stage += 2;
      if (stage >= (uint32_t)kNST) {
        stage -= kNST;
        ph ^= 1;
      }
      if (one) decode(c0, 0, va);
      if (pending) signal();
      // the slot is free once the MMAs of the quad that used it before (qi - kNS) have completed
      if (!__all_sync(0xffffffffu, a_test) && !slot_free()) break;
      tc_fence_after();
      const uint32_t col = a_col + aslot * 128;
      if (one) {
        tc_st16(col, va);
        decode(c0, 1, vb);
        tc_st16(col + 16, vb);
      }
      const bool c_test = !kOdd && mbar_test(bars + 8 * (kBarCFull + stage), ph);
      if (two) {
        decode(c1, 0, va);
        tc_st16(col + 64, va);
        decode(c1, 1, vb);
        tc_st16(col + 80, vb);
      }
      pending = bars + 8 * (kBarAFull + aslot);
      c_ready = __all_sync(0xffffffffu, c_test);
      aslot += 2;
      if (aslot >= (uint32_t)kNS) {
        aslot -= kNS;
        aph ^= 1;
      }
      for (qq += 2; qq >= NQ;) qq -= NQ;
    }
    if (pending) signal();
  } else if (warp >= 20) {
    // ================= epilogue: 16 rows of the expert at a time =================
    const int quarter = warp & 3;
    uint8_t* const ubuf = smem + kOffU;
    volatile int* ep_ok = (volatile int*)(smem + kOffBar + kNumBars * 8 + 16);
    uint32_t li = 0;
    bool ok = true;
    const int e128 = quarter * 32 + lane;
    Tile t_ahead = (int)blockIdx.x < n_items ? p.tiles[blockIdx.x / img.n_mtiles] : Tile{0, 0, 0};
    for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, li++) {
      const Tile t = t_ahead;
      if (it + (int)gridDim.x < n_items) t_ahead = p.tiles[(it + gridDim.x) / img.n_mtiles];
      const int mt = it % img.n_mtiles;
      const uint32_t acc = li & 1, accph = (li >> 1) & 1;
      ok = mbar_wait(bars + 8 * (kBarAccFull + acc), accph, abort_flag, p.status, 8, 256);
      // The four epilogue warps must take the same decision (they meet at named barriers
      // below): publish each warp's result, meet once, and combine.
      ok = __all_sync(0xffffffffu, ok);
      if (lane == 0) ep_ok[(li & 1) * 4 + quarter] = ok ? 1 : 0;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      ok = (ep_ok[(li & 1) * 4] & ep_ok[(li & 1) * 4 + 1] & ep_ok[(li & 1) * 4 + 2] & ep_ok[(li & 1) * 4 + 3]) != 0;
      if (!ok) break;
      tc_fence_after();
      const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + acc * kRows;
      for (int c0 = 0; c0 < t.count; c0 += 16) {
        uint32_t v[16];
        tc_ld16(src + c0, v);
        tc_wait_ld();
        // Results leave through a shared-memory tile [row of the expert][weight row], two of them in turn, so that every
        // global store is a full 16-byte piece of one output row.
        if (UP) {
          // gate rows live in lanes 0..63 (warps 0, 1), the matching up rows in lanes 64..127 (warps 2, 3). Each side
          // hands half of its columns to its partner: gate warps finish rows 0..7, up warps 8..15.
          float* xg = (float*)ubuf;            // [2][8][32] gate values of rows 8..15
          float* xu = xg + 2 * 8 * 32;         // [2][8][32] up values of rows 0..7
          __half* outs = (__half*)(ubuf + 4096 + (c0 & 16) * 128);  // [16][64]
          const int pq = quarter & 1;
          if (quarter < 2) {
#pragma unroll
            for (int j = 0; j < 8; j++) xg[(pq * 8 + j) * 32 + lane] = __uint_as_float(v[8 + j]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) xu[(pq * 8 + j) * 32 + lane] = __uint_as_float(v[j]);
          }
          asm volatile("bar.sync 2, 128;" ::: "memory");
          if (quarter < 2) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const float g = __uint_as_float(v[j]), u = xu[(pq * 8 + j) * 32 + lane];
              outs[j * 64 + pq * 32 + lane] = f16_sat(__fdividef(g, 1.f + __expf(-g)) * u);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const float u = __uint_as_float(v[8 + j]), g = xg[(pq * 8 + j) * 32 + lane];
              outs[(8 + j) * 64 + pq * 32 + lane] = f16_sat(__fdividef(g, 1.f + __expf(-g)) * u);
            }
          }
          asm volatile("bar.sync 3, 128;" ::: "memory");
          const int col = e128 >> 3, seg = e128 & 7;
          if (c0 + col < t.count)
            *(uint4*)(p.out + (size_t)(t.first + c0 + col) * p.out_ld + mt * 64 + seg * 8) = *(const uint4*)(outs + col * 64 + seg * 8);
        } else {
          __half* outs = (__half*)(ubuf + (c0 & 16) * 256);  // [16][128]
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            // two values per conversion; finite values saturate to the fp16 range, NaN stays NaN
            uint32_t h2;
            asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(h2) : "f"(__uint_as_float(v[j + 1])), "f"(__uint_as_float(v[j])));
            outs[j * 128 + e128] = __ushort_as_half((unsigned short)(h2 & 0xFFFFu));
            outs[(j + 1) * 128 + e128] = __ushort_as_half((unsigned short)(h2 >> 16));
          }
          asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int piece = e128 + 128 * k, col = piece >> 4, seg = piece & 15;
            if (c0 + col < t.count)
              *(uint4*)(p.out + (size_t)(t.first + c0 + col) * p.out_ld + mt * 128 + seg * 8) =
                  *(const uint4*)(outs + col * 128 + seg * 8);
          }
        }
      }
      // (the next tile's first chunk writes the buffer that an odd number of chunks left in use: it meets bar 1 first)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (kBarAccEmpty + acc));
    }
  }

  // ---- teardown ----
  if (p.beside && blockIdx.x == 0) pdl_wait();
  __syncthreads();
  if (*abort_flag) {
    // give copies still in flight time to land before the CTA's shared memory goes away
    const unsigned long long t0 = now_ns();
    while (now_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <bool UP, bool DUAL, int FMT>
cudaError_t launch(const TcPlan* plan, const CUtensorMap* m, const Image& img, const Tile* tiles, const int32_t* n_tiles, int max_tiles,
                   __half* out, int out_ld, int32_t* status, cudaStream_t st, bool beside) {
  static OncePerDevice once;  // one per template instance
  if (cudaError_t e = once([] { return cudaFuncSetAttribute(k_expert_few<UP, DUAL, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes); }))
    return e;
  FewParams p{img, tiles, n_tiles, out, out_ld, status, beside ? 1 : 0, plan->margin == 0};
  const long long max_items = (long long)max_tiles * img.n_mtiles;
  const int usable = plan->sms - plan->margin > 1 ? plan->sms - plan->margin : 1;
  const int grid = (int)(max_items < 1 ? 1 : max_items < usable ? max_items : usable);
  // (a margin: no early starts, as in expert_tc.cu)
  return launch_opt(plan->margin == 0, k_expert_few<UP, DUAL, FMT>, dim3(grid), dim3(kThreads), (size_t)kSmemBytes, st, m[0], m[1],
                    m[2], m[3], p);
}

}  // namespace

cudaError_t launch_few(const TcPlan* plan, bool up, bool hidden, const Image& img, const Tile* tiles, const int32_t* n_tiles, int max_tiles,
                       __half* out, int out_ld, int32_t* status, cudaStream_t st, bool beside) {
  const CUtensorMap* m = hidden ? plan->h2 : plan->x2;
  if (up) {
    if (img.fmt == kQ4K) return launch<true, false, kQ4K>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
    if (img.fmt == kQ51) return launch<true, false, kQ51>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
    if (img.dual_book) return launch<true, true, kQ4CP>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
    return launch<true, false, kQ4CP>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
  }
  if (img.fmt == kQ51) return launch<false, false, kQ51>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
  return launch<false, false, kQ4CP>(plan, m, img, tiles, n_tiles, max_tiles, out, out_ld, status, st, beside);
}

}  // namespace b200moe
