// tc_dev.cuh -- device helpers of the grouped GEMMs (expert_tc.cu, expert_few.cu, expert_dense.cu): barriers with
// bounded waits, TMA, tcgen05, and the decoding of packed weights. Included by .cu files only.
#pragma once
#include "kernels.h"
#include "tc.h"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdlib>

namespace b200moe {

struct TcPlan {
  CUtensorMap x[4], h[4];    // activation / hidden maps with boxes of 16, 64, 128, 192 rows of one K block
  CUtensorMap x2[4], h2[4];  // the same with boxes of 16, 32, 48, 64 rows of two K blocks
  CUtensorMap w_dense;       // expanded down weights, boxes of 128 rows of one K block
  int sms = 148;
  int margin = 0;
  long long* trace = nullptr;  // debug timeline of CTA 0 (environment B200MOE_TC_TRACE=<file>)
};

namespace {

constexpr long long kWaitLimitNs = 2000000000ll;  // 2 s: far beyond any legitimate wait

// ---- PTX wrappers ------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// CLUSTER: also what other CTAs of the cluster did before they arrived is seen behind the wait (an arrival of theirs with .release.cluster).
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  // %3: suspend-time hint (ns): sleep in hardware, not in a poll loop
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
  return ok != 0;
}
// One lane of a converged warp. Code around it stays warp-uniform, which lets the compiler
// keep descriptors and addresses in uniform registers instead of converting per instruction.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait. Returns false when the CTA is aborting (this wait or another one gave up).
// `nap_ns` > 0 makes the waiting warp sleep between polls: warps that poll in a tight loop
// take issue slots from the warp that shares their scheduler, and the thread that issues
// the MMAs must not be slowed down by waiters.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int32_t* status, int where, unsigned nap_ns = 0) {
  if (mbar_try<CLUSTER>(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (uint32_t spin = 1;; spin++) {
    if (nap_ns) __nanosleep(nap_ns);
    if (mbar_try<CLUSTER>(bar, parity)) return true;
    if ((spin & 255u) == 0) {
      if (*abort_flag) return false;
      if (now_ns() - t0 > (unsigned long long)kWaitLimitNs) {
        *abort_flag = 1;
        if (atomicCAS(status, 0, 1) == 0) status[1] = where;
        return false;
      }
    }
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor]; fp16 operands, fp32 accumulate.
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
      "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
      "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
      "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major fp16 tile stored as rows of 128 bytes with
// the 128-byte swizzle (what the TMA tensor copy writes): 8-row groups are 1024 bytes
// apart, descriptor version 1 (Blackwell), layout type 2 = 128-byte swizzle.
__device__ __forceinline__ uint64_t b_descriptor(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading-dimension offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride between 8-row groups
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)2 << 61;            // 128-byte swizzle
  return d;
}

// Instruction descriptor: D fp32, A/B fp16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t instr_desc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// fp32 -> fp16, finite values saturating to the fp16 range (as on the GEMV path), NaN staying NaN: one conversion
__device__ __forceinline__ __half f16_sat(float v) {
  unsigned short h;
  asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
  return __ushort_as_half(h);
}

// Per (row, K block) metadata of the source format, as loaded by a dequantising thread.
struct RowMetaTc {
  uint32_t a, b, c, d;
};

// Two fp16 weights from one code byte's table entry `pair` (the two codes as fp16 numbers
// for the GGUF formats, the two code-book values for q4cp) and the group's constants.
template <int FMT>
struct GroupDecode {};
template <>
struct GroupDecode<kQ4CP> {  // w = f16(book) * f16(scale)
  __half2 s2;
  __device__ __forceinline__ void init(const RowMetaTc& m, int h) {
    const uint32_t v = __byte_perm(m.a, 0u, h ? 0x3232u : 0x1010u);  // the half's fp16 scale in both lanes
    s2 = *(const __half2*)&v;
  }
  __device__ __forceinline__ __half2 weight(uint32_t pair, int) const { return __hmul2(*(__half2*)&pair, s2); }
};
template <>
struct GroupDecode<kQ4K> {  // w = (d*sc)*q - (dmin*m), the packed form of src/gguf.h:423-432
  __half2 a2, nb2;
  __device__ __forceinline__ void init(const RowMetaTc& m, int h) {
    const float d = half_bits_to_f32((uint16_t)(m.a & 0xFFFFu)), dmin = half_bits_to_f32((uint16_t)(m.a >> 16));
    const float sc = (float)((m.b >> (16 * h)) & 0xFFu), mn = (float)((m.b >> (16 * h + 8)) & 0xFFu);
    a2 = __float2half2_rn(d * sc);
    nb2 = __float2half2_rn(-(dmin * mn));
  }
  __device__ __forceinline__ __half2 weight(uint32_t pair, int) const { return __hfma2(*(__half2*)&pair, a2, nb2); }
};
template <>
struct GroupDecode<kQ51> {  // w = d*(q + 16*fifth bit) + m, src/gguf.h:360-374
  __half2 d2, m2;
  uint32_t qh;
  __device__ __forceinline__ void init(const RowMetaTc& m, int h) {
    const uint32_t dm = h ? m.c : m.a;
    qh = h ? m.d : m.b;
    d2 = __half2half2(__ushort_as_half((unsigned short)(dm & 0xFFFFu)));
    m2 = __half2half2(__ushort_as_half((unsigned short)(dm >> 16)));
  }
  // byte i of the group holds elements 2i, 2i+1; their fifth bits are bits i, 16 + i of qh:
  // shifted to bits 14 and 30 they read as the fp16 pair (2.0 or 0, 2.0 or 0)
  __device__ __forceinline__ __half2 weight(uint32_t pair, int i) const {
    const uint32_t u = (i <= 14 ? (qh << (14 - i)) : (qh >> 1)) & 0x40004000u;
    const __half2 q5 = __hfma2(*(const __half2*)&u, __float2half2_rn(8.f), *(const __half2*)&pair);
    return __hfma2(q5, d2, m2);
  }
};

}  // namespace

}  // namespace b200moe
