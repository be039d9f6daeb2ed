// expert_gemv.cu -- decode / speculative-verify path (T <= 16): a bandwidth-oriented dequant GEMV. It
// takes the place of k_q4cp_gemv_gg, k_silu_mul_g and k_q4cp_gemv_gd
// (src/gpu/parts/20_kernels_gemv.inc:1607-1764 of the reference): per (token, expert) the 2*mid
// gate/up dot products, SwiGLU, then the d down dot products.
//
// At one token the layer is ~78 MB of 4-bit weights and 138 M multiply-adds. What decides the speed is how many
// shared-memory wavefronts and instructions turn a code into a multiply-add: a multiply-add GEMV on the same
// image (a lane per row, two products per code byte, the activations read by broadcast) spent 37 wavefronts
// on 512 code bytes, of which 16 were table lookups and 16 the activations, and stood at 2.7 TB/s. Here:
//   * mma.m16n8k16 forms the products (exact) and sums (fp32). Its A operand is 16 weight rows: ldmatrix deals the
//     packed codes of a row out to the four lanes of a quad, 8 codes each, a code BYTE becomes an fp16 pair. Scales
//     stay in fp32: no sum runs over two 32-groups. q4cp takes one group per instruction and FOUR or EIGHT rows of an expert per
//     pass over the weights (kMeanRows4 below). Eight rows fill the columns of B; of four, the two groups stand in columns of their
//     own (zeros elsewhere), so that a lane's two columns are the two groups of one row, scaled and added once: half the scale
//     multiplications and partial sums. An instruction adds the same 16 products in either form, and zeros to the other group's
//     columns: the sums are the same to the bit. The GGUF formats take half of each group per instruction, and four rows.
//   * B never moves: a warp owns at most four K blocks (five among longer calls; its slice) of all the rows its team works on, and the
//     activations of a slice are 8 registers per K block and lane.
//   * q4cp: a code byte is decoded by one lookup in a 256-entry half2 table replicated per lane in shared memory
//     (no bank conflicts; a line is 256 bytes, so the address is one byte permute): 32 of the 49 wavefronts per
//     32 x 64 block, which keep the load pipe busy for three quarters of a 13-token launch, its ends included. GGUF: the codes are masked into fp16 bit patterns,
//     code * 2^-24 (denormal, exact), no lookup; 2^24 goes into the fp32 constants. Issue slots bound those.
//   * Weights come by bulk copies into a ring of two or three slots of two K blocks per warp (74 to 123 KB in flight per
//     SM), one copy and one wait per slot; the image keeps a slice's K blocks together (common.cuh).
//   * A unit of work = 32 rows (16 hidden outputs: gate and up rows meet in one warp) over the whole K. The slices
//     leave their sums in shared memory and go on; they take turns at adding up the unit BEFORE, in slice order, so
//     that nobody waits at a barrier. A row's sums depend on nothing but its slice cut, a function of the shape.
//   * Persistent; units are cut into equal contiguous shares per team. The shared expert has CTAs of its own, so
//     that a CTA needs one image's tables.
//   * The gate/up kernel does the routing of a decode call itself (route_block.cuh), every CTA for itself; the last
//     CTA leaves the lists for the kernels behind, the shared expert's CTAs form its gates.
//   * Longer calls with few rows per expert come here with a run list of k_route_scan instead (api.cu, kMinFewWork).
// us of the two kernels, the multiply-add form / this one, 4096 x 1024 with shared expert: T = 1 35 / 28, T = 5
// 120 / 84, T = 13 288 / 191 (gate/up 4.65 TB/s); Q4_K / Q5_1 T = 5 128 / 92 (gate/up 4.6 TB/s, down 4.0: the
// fifth bits); 64 experts of 2048 x 512, 16 tokens (2.2 rows an expert) 90 / 38. One call, T = 1, from the end of the
// kernel in front: routing 4.3 us, first copies and activations 3, gate/up 11, hand-over 2, down 6, combine 5.
#include "kernels.h"
#include "route_block.cuh"

#include <algorithm>

namespace b200moe {

namespace {

constexpr int kWarps = 16;            // compute warps of a CTA
constexpr int kThreads = kWarps * 32;
constexpr int kMaxSubs = 640;         // passes over an expert's weights that a launch takes
constexpr uint32_t kOffLow = 2048;    // the dynamic allocation must start at or below this (its absolute shared address)

// Shared memory map, absolute shared addresses.
// KPW: K blocks of a slice, at most.
// ROWS: rows of an expert that one pass over its weights serves.
template <int FMT, int KPW, int ROWS>
struct Map {
  static_assert(ROWS == 4 || (ROWS == 8 && FMT == kQ4CP), "columns of B");
  static constexpr int kRows = ROWS;
  // Partial-sum buffers of a team, and ring slots per warp: what shared memory holds. For eight rows four buffers and two slots:
  // the buffers let the slices drift further apart, 31.1 against 32.1 us at T = 1, 195.4 / 196.6 at T = 13, than two and
  // three; slices of three K blocks keep two and two.
  static constexpr int kRed = ROWS == 8 && KPW == 3 ? 2 : 4;
  static constexpr int kGroup = KPW >= 4 ? 2 : KPW;             // K blocks per ring slot
  static constexpr int kGroups = (KPW + kGroup - 1) / kGroup;  // slots per unit
  static constexpr uint32_t kLut = kOffLow;  // kQ4CP: 256 lines of {32 lanes x 4 B, first book}{32 x 4 B, second book}
  static constexpr uint32_t kRing = kLut + (FMT == kQ4CP ? 65536u : 0u);
  static constexpr uint32_t kSub = (uint32_t)sub_bytes(FMT), kSlot = kGroup * kSub;
  static constexpr uint32_t kSlots = KPW == 3 || ROWS == 8 ? 2 : 3;
  static constexpr uint32_t kScr = FMT == kQ4K ? 512 : 0;  // per warp: the rows' constants as floats
  static constexpr uint32_t kPart = kRing + kWarps * kSlots * kSlot;          // partial sums [kRed][warp][rows in fours][32 weight rows][4]
  static constexpr uint32_t kBar = kPart + kRed * kWarps * kSubRows * kRows * 4;
  static constexpr uint32_t kBarFull = kBar;                                  // [warp][slot]
  static constexpr uint32_t kBarSum = kBarFull + kWarps * kSlots * 8;         // [team][kRed]: the slices' sums are there
  static constexpr uint32_t kBarFree = kBarSum + kWarps * kRed * 8;           // [team][kRed]: they have been taken
  static constexpr uint32_t kSubs = kBarFree + kWarps * kRed * 8;             // int2 [kMaxSubs]
  static constexpr uint32_t kRowTok = kSubs + kMaxSubs * 8;                   // the token of every routed row, where this kernel routes
  static constexpr uint32_t kScratch = kRowTok + kSmallPairs;
  static constexpr uint32_t kEnd = kScratch + kWarps * kScr;
  static constexpr int kBytes = (int)(kEnd - 1024);
};

struct GemvParams {
  Image img;             // routed experts
  Image img_sh;          // shared expert
  const Run* runs;       // routed runs [n_runs[0]]; the shared run sits at runs[kMaxExperts]
  const int32_t* n_runs;
  int n_sh;              // CTAs 0 .. n_sh-1 work on the shared expert, the others on the routed ones
  int pass0;             // first pass of this launch, of the routed experts and of the shared one alike
  int K;                 // d (gate/up) or mid (down)
  int mid;
  int slices, teams;     // warps that share a unit's K blocks; units in work at a time
  const uint16_t* x;     // gate/up: bf16 [T][d]
  const int32_t* tokidx;
  __half* hid;           // gate/up writes, down reads: fp16 [rows][mid] = silu(gate) * up
  float* out;            // down: pairs fp32 [rows][d], or null:
  __half* out16;         // the same in fp16
  int32_t* status;
  RouteIn route;         // gate/up, fused: the routing is done here (runs, n_runs, tokidx are not read)
  int fused;
  int32_t* ready;        // down: set once the lists are there (null: they were before the gate/up kernel started)
};

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
// the pair table does not change once it is built: these loads may be moved freely
template <uint32_t BASE>
__device__ __forceinline__ uint32_t lut32(uint32_t a) {
  uint32_t v;
  asm("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(BASE));
  return v;
}
__device__ __forceinline__ void ldsm4(uint32_t a, uint32_t* m) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(m[0]), "=r"(m[1]), "=r"(m[2]), "=r"(m[3]) : "r"(a) : "memory");
}
// c += a (16 rows x 16) * b (16 x 8), fp16 operands, fp32 sums
__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16816_first(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
  return ok != 0;
}
// Bounded wait (2 s), all lanes of a warp. After one that gave up the warp waits no more: what it computes is
// void, the status word tells.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, int32_t* status, int where) {
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  for (;;) {
    if (mbar_try(bar, parity)) return false;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    if (t - t0 > 2000000000ull) {
      if (status && atomicCAS(status, 0, 8) == 0) status[1] = where;
      return true;
    }
  }
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, bool& dead, int32_t* status, int where) {
  if (!mbar_try(bar, parity) && !dead) dead = mbar_wait_slow(bar, parity, status, where);
}

// finite values saturate to the fp16 range, NaN stays NaN
__device__ __forceinline__ float sat_f16(float v) { return v != v ? v : fminf(fmaxf(v, -65504.f), 65504.f); }
__device__ __forceinline__ uint32_t bf16x2_to_f16x2(uint32_t w) {
  const __half2 h = __floats2half2_rn(sat_f16(__uint_as_float(w << 16)), sat_f16(__uint_as_float(w & 0xFFFF0000u)));
  return *(const uint32_t*)&h;
}

template <bool UP, int FMT, int KPW, int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
k_gemv(const __grid_constant__ GemvParams p) {
  using M = Map<FMT, KPW, ROWS>;
  constexpr bool kHalves = ROWS == 4;  // the two groups of a K block in columns of their own
  constexpr int kRows = M::kRows, kRed = M::kRed;
  extern __shared__ __align__(16) uint8_t gsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  {
    // the map stands at fixed absolute shared addresses: a launch whose dynamic allocation does not
    // cover it is refused (uniform for the grid; the host sizes it)
    const uint32_t dyn0 = (uint32_t)__cvta_generic_to_shared(gsm);
    uint32_t dyn_size;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
    if (dyn0 > kOffLow || dyn0 + dyn_size < M::kEnd) return;
  }
  const bool sh = (int)blockIdx.x < p.n_sh;
  const Image& im = sh ? p.img_sh : p.img;
  // ---- set-up that needs weights only, nothing an earlier kernel of the stream writes ----
  if (tid < kWarps * (int)M::kSlots) mbar_init(M::kBarFull + tid * 8, 1);
  if (tid < kWarps * kRed) {
    mbar_init(M::kBarSum + tid * 8, p.slices);
    mbar_init(M::kBarFree + tid * 8, 1);
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (FMT == kQ4CP) {
    // entry e = (f16(book[e & 15]), f16(book[e >> 4])); warp w writes the 16 lines whose high code is w
    for (int b = 0; b < (UP && im.dual_book ? 2 : 1); b++) {
      const uint32_t hi16 = (uint32_t)__half_as_ushort(__float2half_rn(__ldg(im.book + b * 16 + warp))) << 16;
      const uint32_t mine = (uint32_t)__half_as_ushort(__float2half_rn(__ldg(im.book + b * 16 + (lane & 15))));
      const uint32_t dst = M::kLut + (uint32_t)(warp * 16 * 256 + b * 128 + lane * 4);
#pragma unroll
      for (int c = 0; c < 16; c++) sts32(dst + c * 256, hi16 | __shfl_sync(0xffffffffu, mine, c));
    }
  }
  int n_subs;
  auto put_pass = [&](int i, int expert, int first, int count) {
    i -= p.pass0;
    if ((unsigned)i < (unsigned)kMaxSubs) {
      sts32(M::kSubs + i * 8, (uint32_t)expert | (uint32_t)count << 16);
      sts32(M::kSubs + i * 8 + 4, (uint32_t)first);
    }
  };
  uint8_t* const smem = gsm - (uint32_t)__cvta_generic_to_shared(gsm);  // smem + A is the generic pointer of absolute shared address A
  uint8_t* const row_token = smem + M::kRowTok;
  const int KB = im.n_kblocks, ash = im.act_shift;
  const int slice = warp % p.slices, team = warp / p.slices;
  const int kb0 = slice * KPW, nk = min(KPW, KB - kb0);
  // Activations of the slice, B operands. Eight rows: lane (g, t) holds row g, elements 8t .. 8t+7 of both halves of every
  // K block. Four: row g >> 1, half g & 1, in bv for half 0 and in bw for half 1, zeros in the other.
  uint32_t bv[KPW][4], bw[KPW][4];
  float xs[KPW][2];             // GGUF: sums of the activations of row t, halves 0 and 1
  auto load_rows = [&](bool live, size_t row) {
    auto load8 = [&](int i, int h, uint32_t* v) {
      uint4 u = make_uint4(0, 0, 0, 0);
      if (live && i < nk) {
        const size_t o = row * p.K + (size_t)((kb0 + i) >> ash) * kTileK + h * 32 + t * 8;
        u = UP ? __ldg((const uint4*)(p.x + o)) : *(const uint4*)(p.hid + o);
      }
      v[0] = UP ? bf16x2_to_f16x2(u.x) : u.x;
      v[1] = UP ? bf16x2_to_f16x2(u.y) : u.y;
      v[2] = UP ? bf16x2_to_f16x2(u.z) : u.z;
      v[3] = UP ? bf16x2_to_f16x2(u.w) : u.w;
    };
#pragma unroll
    for (int i = 0; i < KPW; i++) {
      if (!kHalves) {
        load8(i, 0, bv[i]);
        load8(i, 1, bw[i]);
      } else {
        uint32_t v[4];
        load8(i, g & 1, v);
        if (FMT == kQ4K) {  // pairs of elements q and q + 4
          const uint32_t w0 = v[0], w1 = v[1];
          v[0] = __byte_perm(w0, v[2], 0x5410);
          v[1] = __byte_perm(w0, v[2], 0x7632);
          v[2] = __byte_perm(w1, v[3], 0x5410);
          v[3] = __byte_perm(w1, v[3], 0x7632);
        }
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          bv[i][q] = (g & 1) ? 0u : v[q];
          bw[i][q] = (g & 1) ? v[q] : 0u;
          if (FMT != kQ4CP) mma16816(c, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, bv[i][q], bw[i][q]);
        }
        xs[i][0] = c[0];
        xs[i][1] = c[1];
      }
    }
  };
  if (UP) pdl_wait();
  // One token: its activations serve every row of every pass (a caller's ids may repeat), and travel while the routing runs.
  const bool one = UP && p.fused && p.route.T == 1;
  if (one) load_rows(true, 0);
  if (UP && p.fused) {
    // ---- routing (route_block.cuh), by every CTA of the routed experts for itself; the last one, whose share is
    // never the larger, leaves the lists and weights for the kernels behind. Its scratch is the place of the partial sums, which come later ----
    static_assert(kSmallPairs <= kMaxSubs, "a call that is routed here fits one launch");
    static_assert(kRouteBlockBytes <= kRed * kWarps * kSubRows * kRows * 4, "the routing's scratch");
    if (sh) {
      n_subs = (p.route.T + kRows - 1) / kRows;
      if (tid < n_subs) put_pass(tid, 0, p.route.T * p.route.k + tid * kRows, min(kRows, p.route.T - tid * kRows));
    } else {
      n_subs = route_block(p.route, *(RouteBlock*)(smem + M::kPart), blockIdx.x == gridDim.x - 1, kRows, row_token,
                           [&](int expert, int first, int count, int at) {
                             for (int i = 0; i * kRows < count; i++) put_pass(at + i, expert, first + i * kRows, min(kRows, count - i * kRows));
                           });
    }
    __syncthreads();
    if (blockIdx.x == gridDim.x - 1 && tid == 0) {
      __threadfence();
      asm volatile("st.release.gpu.global.b32 [%0], 1;" ::"l"(p.route.rb.ready) : "memory");
    }
    pdl_trigger();  // (behind the flag: the down kernel starts when every CTA has come here)
  } else {
    if (UP) pdl_trigger();
    // ---- passes: every expert's rows, kRows at a time ----
    // The down kernel reads the run list before its wait: the routing kernel was complete before any CTA of the
    // gate/up kernel triggered, or, where that kernel routes, the flag tells.
    __shared__ int s_cnt[kWarps];
    if (!UP && p.ready) {
      if (tid == 0) {
        unsigned long long t0 = 0, now;
        int v;
        for (;;) {
          asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p.ready) : "memory");
          if (v) break;
          asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          if (now - t0 > 2000000000ull) {
            if (p.status && atomicCAS(p.status, 0, 8) == 0) p.status[1] = 23;
            break;
          }
        }
      }
      __syncthreads();
    }
    const int n_runs = sh ? 1 : min(__ldcg(p.n_runs), kThreads);
    Run run{0, 0, 0};
    if (tid < n_runs) {
      const int32_t* r = (const int32_t*)(p.runs + (sh ? kMaxExperts : tid));
      run = Run{__ldcg(r), __ldcg(r + 1), __ldcg(r + 2)};
    }
    const int c = (run.count + kRows - 1) / kRows;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_cnt[warp] = incl;
    __syncthreads();
    int before = incl - c;
    n_subs = 0;
    for (int w = 0; w < kWarps; w++) {
      const int v = s_cnt[w];
      if (w < warp) before += v;
      n_subs += v;
    }
    n_subs = min(max(n_subs - p.pass0, 0), kMaxSubs);
    for (int i = 0; i < c; i++) put_pass(before + i, run.expert, run.first + i * kRows, min(kRows, run.count - i * kRows));
    __syncthreads();
  }
  // ---- this team's share: units c0 .. c1-1 of all passes. A unit = one sub-block column, 32 tile rows over the whole K ----
  const int upr = im.n_mtiles * 4;  // units of a pass
  int c0, n_units;
  {
    const int total = n_subs * upr;
    const int n_ct = sh ? p.n_sh : (int)gridDim.x - p.n_sh, ci = sh ? (int)blockIdx.x : (int)blockIdx.x - p.n_sh;
    const int nt = n_ct * p.teams, ti = ci * p.teams + team;
    const int base = total / nt, rem = total % nt;
    c0 = ti * base + min(ti, rem);
    n_units = base + (ti < rem ? 1 : 0);
  }
  if (team >= p.teams) n_units = 0;
  // ---- the copy stream: a slot = one group of K blocks of a unit, M::kSlots groups ahead ----
  const uint32_t ring = M::kRing + (uint32_t)warp * M::kSlots * M::kSlot, full = M::kBarFull + (uint32_t)warp * M::kSlots * 8;
  int q_left = n_units, q_g = 0, q_sub = c0 / upr, q_j = c0 % upr;
  uint32_t q_slot = 0;
  const uint32_t unit_b = (uint32_t)KB * M::kSub;
  const uint8_t* q_ptr;  // the slice's first K block of the unit at hand: the units of an expert follow one another
  auto q_pass = [&]() {
    const uint32_t e = lds32(M::kSubs + q_sub * 8) & 0xFFFFu;
    q_ptr = im.data + ((size_t)e * upr + q_j) * unit_b + (uint32_t)kb0 * M::kSub;
  };
  if (n_units > 0) q_pass();
  auto issue = [&]() {
    if (q_left > 0) {
      if (lane == 0) {
        const uint32_t bar = full + q_slot * 8;
        const uint32_t bytes = min(M::kGroup, nk - q_g * M::kGroup) * M::kSub;  // > 0: groups without K blocks are stepped over
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         ring + q_slot * M::kSlot), "l"(q_ptr + q_g * M::kSlot), "r"(bytes), "r"(bar)
                     : "memory");
      }
      q_slot = q_slot + 1 == M::kSlots ? 0 : q_slot + 1;
      if (M::kGroups > 1 && q_g + 1 < M::kGroups && (q_g + 1) * M::kGroup < nk) {
        q_g++;
      } else {
        q_g = 0;
        q_left--;
        q_j++;
        q_ptr += unit_b;
        if (q_j == upr) {
          q_j = 0;
          q_sub++;
          if (q_left > 0) q_pass();
        }
      }
    }
  };
  for (uint32_t s = 0; s < M::kSlots; s++) issue();
  if (!UP) {
    // The launch behind comes behind this wait: the combine of a decode call reads its lists before its own wait, and
    // a tensor-core launch may run beside this one.
    pdl_wait();
    pdl_trigger();
  }
  if (UP && p.fused && sh && p.route.gate_w) {
    gate_block(p.route, blockIdx.x, p.n_sh, tid, (double*)(smem + M::kPart), [] { __syncthreads(); });
    __syncthreads();  // (its scratch is the place of the partial sums)
  }
  if (n_units == 0) return;

  bool dead = false, lost = false;  // a wait for the team, for the warp's own copies gave up
  uint32_t c_slot = 0, c_ph = 0;
  int sub = c0 / upr, j = c0 % upr, cnt = 0, first = 0;
  bool fresh = true;
  const uint32_t lut_a = (uint32_t)lane * 4, lut_b = lut_a + (UP && im.dual_book ? 128u : 0u);
  const uint32_t lane_src = (uint32_t)(lane >> 4) * kHalfBytes + (uint32_t)(lane & 15) * 16;
  const uint32_t part0 = M::kPart + (uint32_t)(team * p.slices) * (kSubRows * kRows * 4);
  constexpr uint32_t kPartBuf = kWarps * kSubRows * kRows * 4;
  const uint32_t bar_sum = M::kBarSum + team * kRed * 8, bar_free = M::kBarFree + team * kRed * 8;
  // adds the slices of unit n (its number in this team's share) in slice order and writes its results
  auto finish = [&](int n, int uj, int ucnt, int ufirst) {
    const uint32_t b = n & (kRed - 1);
    mbar_wait(bar_sum + b * 8, (n / kRed) & 1, dead, p.status, 22);
    float tot[kRows];
    const uint32_t a = part0 + b * kPartBuf + lane * 16;
#pragma unroll
    for (int pl = 0; pl < kRows; pl += 4) {
      tot[pl] = tot[pl + 1] = tot[pl + 2] = tot[pl + 3] = 0.f;
      if (pl < ucnt) {
#pragma unroll 4
        for (int s = 0; s < p.slices; s++) {
          const uint4 v = lds128(a + s * (kSubRows * kRows * 4) + pl * (kSubRows * 4));
          tot[pl] += __uint_as_float(v.x);
          tot[pl + 1] += __uint_as_float(v.y);
          tot[pl + 2] += __uint_as_float(v.z);
          tot[pl + 3] += __uint_as_float(v.w);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_free + b * 8);
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      if (r < ucnt) {
        if (UP) {
          const float up = __shfl_down_sync(0xffffffffu, tot[r], 16);
          if (lane < 16)
            p.hid[(size_t)(ufirst + r) * p.mid + uj * 16 + lane] = __float2half_rn(sat_f16(silu_f32(tot[r]) * up));
        } else {
          const size_t o = (size_t)(ufirst + r) * (upr * kSubRows) + uj * kSubRows + lane;
          if (p.out) p.out[o] = tot[r];
          else p.out16[o] = __float2half_rn(sat_f16(tot[r]));
        }
      }
    }
  };
  constexpr int kAcc = kRows / 4;  // activation rows of a lane: t, or 2t and 2t + 1
  // one K block (number i of the slice) of a unit: 32 rows x 64 columns
  auto item = [&](int i, uint32_t s0, float (&acc)[2][2][kAcc]) {
    uint32_t m[2][4];
    ldsm4(s0 + lane_src, m[0]);
    ldsm4(s0 + lane_src + 256, m[1]);
    float k[2][2][4];  // constants of the lane's rows: factors of the two halves' sums (and of the activations' sums)
    if (FMT == kQ4K) {
      // a lane turns one row's constants into floats, all lanes pick up theirs
      const uint32_t sa = M::kScratch + warp * 512;
      const uint2 v = lds64(s0 + kSubCodes + lane * 8);
      const float2 dd = __half22float2(*(const __half2*)&v.x);
      // {sc0, m0, sc1, m1} as fp16 1024 + value, then exactly the values
      const uint32_t u0 = __byte_perm(v.y, 0x64646464u, 0x4240), u1 = __byte_perm(v.y, 0x64646464u, 0x4341);
      const __half2 k1024 = __float2half2_rn(1024.f);
      const float2 sc = __half22float2(__hsub2(*(const __half2*)&u0, k1024)), mn = __half22float2(__hsub2(*(const __half2*)&u1, k1024));
      const float ds = dd.x * 16777216.f;  // the codes stand as code * 2^-24
      __syncwarp();
      asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(sa + lane * 16), "f"(ds * sc.x), "f"(ds * sc.y), "f"(-dd.y * mn.x), "f"(-dd.y * mn.y) : "memory");
      __syncwarp();
#pragma unroll
      for (int b = 0; b < 2; b++)
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const uint4 w = lds128(sa + (uint32_t)(b * 16 + r * 8 + g) * 16);
          k[b][r][0] = __uint_as_float(w.x); k[b][r][1] = __uint_as_float(w.y); k[b][r][2] = __uint_as_float(w.z); k[b][r][3] = __uint_as_float(w.w);
        }
    }
    uint32_t f[2][4];
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t ma = s0 + kSubCodes + (uint32_t)(b * 16 + r * 8 + g) * meta_row_bytes(FMT);
        if (FMT == kQ4CP) {
          const uint32_t v = lds32(ma);
          const float2 s = __half22float2(*(const __half2*)&v);
          k[b][r][0] = s.x; k[b][r][1] = s.y;
        } else if (FMT == kQ51) {
          const uint4 v = lds128(ma);
          const float2 e0 = __half22float2(*(const __half2*)&v.x), e1 = __half22float2(*(const __half2*)&v.z);
          k[b][r][0] = e0.x * 16777216.f; k[b][r][1] = e1.x * 16777216.f; k[b][r][2] = e0.y; k[b][r][3] = e1.y;
          // this lane's eight fifth bits of the row's two halves to bits 0..3 and 16..19
          f[b][r] = v.y >> (4 * t);
          f[b][2 + r] = v.w >> (4 * t);
        }
      }
#pragma unroll
    for (int b = 0; b < 2; b++) {
      if (FMT == kQ4CP) {
        float c[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          // the half's products: K slots 2t, 2t+1 are the codes of byte 2q, slots 2t+8, 2t+9 those of byte 2q+1
#pragma unroll
          for (int q = 0; q < 2; q++) {
            uint32_t a[4];
#pragma unroll
            for (int i4 = 0; i4 < 4; i4++)
              a[i4] = lut32<M::kLut>(__byte_perm(m[b][2 * h + (i4 & 1)], b ? lut_b : lut_a, 0x5504 | (2 * q + (i4 >> 1)) << 4));
            const uint32_t b0 = h ? bw[i][2 * q] : bv[i][2 * q], b1 = h ? bw[i][2 * q + 1] : bv[i][2 * q + 1];
            if (q == 0 && !(kHalves && h == 1)) mma16816_first(c, a[0], a[1], a[2], a[3], b0, b1);
            else mma16816(c, a[0], a[1], a[2], a[3], b0, b1);
          }
          if (!kHalves) {
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
              for (int w = 0; w < kAcc; w++) acc[b][r][w] = fmaf(k[b][r][h], c[2 * r + w], acc[b][r][w]);
          }
        }
        if (kHalves) {
#pragma unroll
          for (int r = 0; r < 2; r++) acc[b][r][0] = fmaf(k[b][r][1], c[2 * r + 1], fmaf(k[b][r][0], c[2 * r], acc[b][r][0]));
        }
      } else {
        float c[4], c16[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t a[4];
#pragma unroll
          for (int h = 0; h < 4; h++) {
            if (FMT == kQ4K) {
              // codes q and q + 4 of the word as the fp16 pair code * 2^-24, for odd q 16 times that (denormal numbers: exact, also in the products)
              a[h] = (q & 2 ? m[b][h] >> 8 : m[b][h]) & (q & 1 ? 0x00F000F0u : 0x000F000Fu);
            } else {
              // the two codes of byte q as the fp16 pair code * 2^-24
              a[h] = __byte_perm(m[b][h], m[b][h] >> 4, q | (4 + q) << 8) & 0x000F000Fu;
              a[h] |= (f[b][h] << (4 - q)) & 0x00100010u;
            }
          }
          float* cc = FMT == kQ4K && (q & 1) ? c16 : c;
          if (q == 0 || (FMT == kQ4K && q == 1)) mma16816_first(cc, a[0], a[1], a[2], a[3], bv[i][q], bw[i][q]);
          else mma16816(cc, a[0], a[1], a[2], a[3], bv[i][q], bw[i][q]);
        }
        if (FMT == kQ4K) {
#pragma unroll
          for (int h = 0; h < 4; h++) c[h] = fmaf(c16[h], 0.0625f, c[h]);
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
          acc[b][r][0] = fmaf(k[b][r][1], c[2 * r + 1], fmaf(k[b][r][0], c[2 * r], acc[b][r][0]));
          acc[b][r][0] = fmaf(k[b][r][3], xs[i][1], fmaf(k[b][r][2], xs[i][0], acc[b][r][0]));
        }
      }
    }
  };
  int pj = 0, pcnt = 0, pfirst = 0, turn = 0;
  for (int n = 0; n <= n_units; n++) {
   if (n < n_units) {
    if (fresh) {
      fresh = false;
      const uint2 e = lds64(M::kSubs + sub * 8);
      cnt = (int)(e.x >> 16);
      first = (int)e.y;
      const int at = kHalves ? g >> 1 : g;
      const bool live = at < cnt;
      size_t row = first + at;
      if (UP && live) row = !p.fused ? p.tokidx[row] : sh ? row - p.route.T * p.route.k : row_token[row];
      if (!live) row = 0;
      if (!one) load_rows(live, row);
    }
    float acc[2][2][kAcc] = {};  // [16-row block][weight row g, g + 8][activation rows of the lane]
#pragma unroll
    for (int gi = 0; gi < M::kGroups; gi++) {
      if (gi * M::kGroup < nk) {
        mbar_wait(full + c_slot * 8, c_ph, lost, p.status, 20);
        const uint32_t slot0 = ring + c_slot * M::kSlot;
#pragma unroll
        for (int ii = 0; ii < M::kGroup; ii++) {
          const int i = gi * M::kGroup + ii;
          if (i < KPW && i < nk) item(i, slot0 + ii * M::kSub, acc);
        }
        __syncwarp();
        issue();  // the slot has been read
        c_slot++;
        if (c_slot == M::kSlots) {
          c_slot = 0;
          c_ph ^= 1;
        }
      }
    }
    // ---- the slice's sums of this unit ----
    const uint32_t b = n & (kRed - 1);
    if (n >= kRed) mbar_wait(bar_free + b * 8, ((n / kRed) & 1) ^ 1, dead, p.status, 21);
    if (t * kAcc < cnt) {
      const uint32_t a = part0 + b * kPartBuf + (uint32_t)slice * (kSubRows * kRows * 4) + (uint32_t)((t * kAcc) >> 2) * (kSubRows * 16) +
                         (uint32_t)g * 16 + ((t * kAcc) & 3) * 4;
#pragma unroll
      for (int bb = 0; bb < 2; bb++)
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
          for (int w = 0; w < kAcc; w++) sts32(a + (bb * 16 + r * 8) * 16 + w * 4, __float_as_uint(acc[bb][r][w]));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_sum + b * 8);
   }
    // the slices take turns at finishing the unit before this one, whose last sums have come in meanwhile
    if (n > 0) {
      if (turn == slice) finish(n - 1, pj, pcnt, pfirst);
      turn = turn + 1 == p.slices ? 0 : turn + 1;
    }
    pj = j;
    pcnt = cnt;
    pfirst = first;
    if (++j == upr) {
      j = 0;
      sub++;
      fresh = true;
    }
  }
}

template <bool UP, int FMT, int KPW, int ROWS>
cudaError_t launch_gemv(const GemvParams& p, cudaStream_t st) {
  constexpr int smem = Map<FMT, KPW, ROWS>::kBytes;
  static OncePerDevice once;
  if (cudaError_t e = once([] { return cudaFuncSetAttribute(k_gemv<UP, FMT, KPW, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); }))
    return e;
  int sms = 0;
  if (cudaError_t e = sm_count(&sms)) return e;
  return launch_pdl(k_gemv<UP, FMT, KPW, ROWS>, dim3(sms), dim3(kThreads), (size_t)smem, st, p);
}

// One launch for the passes pass0 .. pass0 + kMaxSubs - 1.
template <bool UP, int FMT, int ROWS>
cudaError_t launch_one(GemvParams& p, bool decode, cudaStream_t st) {
  const int KB = p.img.n_kblocks;
  // K blocks per warp: what leaves the fewest of the 16 warps idle or short of a block; in decode calls longer slices, whose chain is longer, only where
  // they put an eighth more to work (K = 384: two slices of three instead of three of two, 16 against 15 warps: 26.6 against 25.9 us). (At
  // K = 1280 ten slices of two leave six warps idle: five of four, three units at a time, 58.4 -> 52.2 us of a 13-token call of
  // 1280 x 768, 74.7 -> 64.5 of 1280 x 1024; K = 1536 8 slices of three instead of 12 of two, 44.0 -> 39.9.) Five only for eight
  // rows per pass among longer calls: 500 tokens of 2560 x 640 380 -> 370 us, 100 tokens 329 -> 316; with four rows, whose blocks are cheaper, 2560 x 640
  // is level and 2304 x 1024 loses 4 %. The cut decides the order of the sums: one of the shape alone in all decode calls.
  const bool longer = ROWS == 8 && !decode;
  int kpw = 0, best = 0;
  for (int n = 2; n <= (longer ? 5 : 4); n++) {
    const int slices = (KB + n - 1) / n;
    if (slices > kWarps) continue;
    const int busy = KB * (kWarps / slices) * (60 / n);  // K blocks at work of 16 * n, times 960
    if (longer ? busy > best : 8 * busy >= 9 * best) best = busy, kpw = n;
  }
  if (kpw == 0) return cudaErrorInvalidValue;
  p.slices = (KB + kpw - 1) / kpw;
  p.teams = kWarps / p.slices;
  if constexpr (ROWS == 8)
    if (kpw == 5) return launch_gemv<UP, FMT, 5, ROWS>(p, st);
  if (kpw == 4) return launch_gemv<UP, FMT, 4, ROWS>(p, st);
  if (kpw == 3) return launch_gemv<UP, FMT, 3, ROWS>(p, st);
  return launch_gemv<UP, FMT, 2, ROWS>(p, st);
}

// Passes that the host cannot count take as many launches as could be needed (a call of up to 16 tokens: one). Each
// waits for the one before; those beyond the last pass end at once.
template <bool UP, int FMT, int ROWS>
cudaError_t launch_fmt(GemvParams& p, int T, int max_passes, bool decode, int* launches, cudaStream_t st) {
  if (p.n_sh > 0) max_passes = std::max(max_passes, (T + ROWS - 1) / ROWS);
  for (p.pass0 = 0; p.pass0 == 0 || p.pass0 < max_passes; p.pass0 += kMaxSubs) {
    if (cudaError_t e = launch_one<UP, FMT, ROWS>(p, decode, st)) return e;
    ++*launches;
  }
  return cudaSuccess;
}

// CTAs for the shared expert: its share of the passes that T tokens with even routing make. (Fewer routed
// passes than that only leave the routed CTAs idle a little earlier.)
int shared_ctas(int T, int k, int E, int rows) {
  const double idle = 1.0 - (double)k / E;
  double unused = 1.0;
  for (int i = 0; i < T; i++) unused *= idle;
  const double routed = E * (1.0 - unused) * 1.02, shared = (T + rows - 1) / rows;
  const int n = (int)(148.0 * shared / (routed + shared)) + 1;  // rounded up: a CTA less would be the one that all wait for
  return n > 74 ? 74 : n;
}

// Rows per pass of a decode call: eight cost an expert with up to four rows 1 to 5 % of the call more, four cost one with five to eight a second pass.
// us of a call, four / eight: 512 experts of 4096 x 1024 + shared, top-10, T = 1 / 5 / 13 30.2 / 30.9, 83.1 / 87.3, 191.3 / 194.4; 512 of 2560 x
// 640 + shared, 5 / 13 44.8 / 46.0, 85.1 / 88.4; 64 of 2048 x 512, top-8, 5 / 16 27.4 / 27.2, 38.1 / 38.6. Few experts of 4096 x 1024: 2.25 rows each
// on average (top-4 of 16 and top-8 of 32 at T = 9) 37.0 / 37.6 and 57.8 / 59.1, 3.25 (T = 13) 42.4 / 39.1 and 67.9 / 61.8, 4.5 (top-8 of 16 at
// T = 9) 50.0 / 40.8, 8 (T = 16) 68.7 / 51.8. The line lies at 11/4; both forms give the same bits.
constexpr int kMeanRows4 = 11;
int decode_rows(int fmt, int T, int k, int E) { return fmt == kQ4CP && T > 4 && 4ll * T * k > (long long)kMeanRows4 * E ? 8 : 4; }

}  // namespace

int gemv_max_runs() { return 192; }
int gemv_rows(int fmt) { return fmt == kQ4CP ? 8 : 4; }
int gemv_passes(int fmt, int T, int k, int E) {
  const int rows = decode_rows(fmt, T, k, E), runs = T * k < E ? T * k : E;
  return (T * k + runs * (rows - 1)) / rows;
}
int gemv_max_k() { return kWarps * 4 * kTileK; }
int gemv_max_mid() { return kWarps / 2 * 4 * kTileK; }

cudaError_t launch_up_gemv(const Image& img, const Image* img_sh, const void* x_bf16, int T, int k, int E, int d, int mid,
                           const int32_t* tokidx, const Run* runs, const int32_t* n_runs,
                           int max_passes, bool decode, __half* hid16, int32_t* status, const RouteIn* route, int* launches,
                           cudaStream_t st) {
  GemvParams p{};
  p.img = img;
  const int rows = decode ? decode_rows(img.fmt, T, k, E) : gemv_rows(img.fmt);
  if (img_sh) p.img_sh = *img_sh, p.n_sh = shared_ctas(T, k, E, rows);
  p.runs = runs; p.n_runs = n_runs; p.K = d; p.mid = mid;
  p.x = (const uint16_t*)x_bf16; p.tokidx = tokidx; p.hid = hid16; p.status = status;
  if (route) p.route = *route, p.fused = 1;
  if (img.fmt == kQ4K) return launch_fmt<true, kQ4K, 4>(p, T, max_passes, decode, launches, st);
  if (img.fmt == kQ51) return launch_fmt<true, kQ51, 4>(p, T, max_passes, decode, launches, st);
  if (rows == 4) return launch_fmt<true, kQ4CP, 4>(p, T, max_passes, decode, launches, st);
  return launch_fmt<true, kQ4CP, 8>(p, T, max_passes, decode, launches, st);
}

cudaError_t launch_down_gemv(const Image& img, const Image* img_sh, const __half* hid16, int T, int k, int E, int d, int mid,
                             const Run* runs, const int32_t* n_runs, int max_passes, bool decode, void* pairs, bool pairs_f16, int32_t* status,
                             int32_t* ready, int* launches, cudaStream_t st) {
  GemvParams p{};
  p.img = img;
  const int rows = decode ? decode_rows(img.fmt, T, k, E) : gemv_rows(img.fmt);
  if (img_sh) p.img_sh = *img_sh, p.n_sh = shared_ctas(T, k, E, rows);
  p.runs = runs; p.n_runs = n_runs; p.K = mid; p.mid = mid;
  p.hid = const_cast<__half*>(hid16);
  if (pairs_f16) p.out16 = (__half*)pairs; else p.out = (float*)pairs;
  p.status = status; p.ready = ready;
  if (img.fmt == kQ4K) return launch_fmt<false, kQ4K, 4>(p, T, max_passes, decode, launches, st);
  if (img.fmt == kQ51) return launch_fmt<false, kQ51, 4>(p, T, max_passes, decode, launches, st);
  if (rows == 4) return launch_fmt<false, kQ4CP, 4>(p, T, max_passes, decode, launches, st);
  return launch_fmt<false, kQ4CP, 8>(p, T, max_passes, decode, launches, st);
}

}  // namespace b200moe
