// PTX wrappers and epilogue arithmetic shared by the tcgen05 kernels (sm_100a): mbarriers, TMA loads, tensor
// memory, the MMA issue, shared-memory and instruction descriptors, and the running (max, argmax) fold over
// accumulator columns.
#pragma once

#include <cuda.h>

#include "lik_common.cuh"

namespace lik {
namespace {

constexpr int TILE_M = 128;                   // accumulator rows (TMEM lanes) of every MMA

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same with a hint how long the hardware may keep the thread suspended.
__device__ __forceinline__ bool mbar_try_wait_long(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(20000)
      : "memory");
  return ok != 0;
}
constexpr long long WAIT_LIMIT_CYCLES = 4000000000ll;  // default limit of a wait: about 2 s at 2 GHz

// What the bounded waits of a CTA share, in shared memory.
struct WaitCtl {
  volatile int abort_flag;
  volatile int progress;  // counted up by a warp that is busy for longer than a wait's limit may be: who waits for it begins anew
  long long limit;
  __device__ __forceinline__ void init(long long cycles = WAIT_LIMIT_CYCLES) {
    abort_flag = progress = 0;
    limit = cycles;
  }
};
// Bounded wait of a whole warp; the lanes leave together, with one answer.  False: the CTA is aborting.  (No suspension hint: a warp
// that it puts to sleep comes back late, 642 us against 587 in the compressed-index kernel.)
// The flag and the clock are looked at after every sixteenth question: what a waiting warp issues, others cannot.
__device__ __forceinline__ bool wait_bar_all(unsigned long long* bar, uint32_t parity, WaitCtl* ctl, int* status) {
  const uint32_t b = smem_u32(bar);
  if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
  long long t0 = clock64();
  int seen = 0;
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i)
      if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
    if (clock64() - t0 > ctl->limit) {
      const int now = ctl->progress;
      if (now == seen) {
        ctl->abort_flag = 1;
        if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
      }
      seen = now;
      t0 = clock64();
    }
    if (__any_sync(0xffffffffu, ctl->abort_flag != 0)) return false;
  }
}
// generic-proxy writes to shared memory become visible to the async proxy (the tensor core's operand reads)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// untiled bulk copy global -> shared (16-byte aligned on both sides, a multiple of 16 bytes), completing on an mbarrier
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Both operand descriptors share their upper word (stride, version, swizzle mode); only the 14-bit
// start-address field in the lower word moves, so the issuer carries 32-bit values and the 64-bit
// descriptors are put together next to the instruction.
template <bool FP8>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                       uint32_t accumulate) {
  if (FP8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// The same with A in tensor memory: lane = row, eight columns per 32 bytes of K.
template <bool FP8>
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
  if (FP8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// 128 rows x 32 bytes of a K-major operand tile in shared memory -> 128 lanes x 8 columns of tensor memory, as tc_mma_ts reads A
__device__ __forceinline__ void tc_copy_128x256b(uint32_t taddr, uint32_t desc_lo, uint32_t desc_hi) {
  asm volatile("{\n\t.reg .b64 d;\n\tmov.b64 d, {%1, %2};\n\ttcgen05.cp.cta_group::1.128x256b [%0], d;\n\t}" ::"r"(taddr), "r"(desc_lo), "r"(desc_hi) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns of TMEM -> 32 registers per thread.  The load is
// asynchronous: the registers may only be read after tmem_ld_wait(), which takes them as in/out
// operands so that no use can be scheduled ahead of it.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, float (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(float (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15]), "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]), "+f"(v[22]), "+f"(v[23]), "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]), "+f"(v[29]), "+f"(v[30]), "+f"(v[31]) : : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// maximum of 32 values as a shallow tree of independent 3-input max operations
__device__ __forceinline__ float max32(const float (&v)[32]) {
  float a0 = max3(v[0], v[1], v[2]), a1 = max3(v[3], v[4], v[5]), a2 = max3(v[6], v[7], v[8]);
  float a3 = max3(v[9], v[10], v[11]), a4 = max3(v[12], v[13], v[14]), a5 = max3(v[15], v[16], v[17]);
  float a6 = max3(v[18], v[19], v[20]), a7 = max3(v[21], v[22], v[23]), a8 = max3(v[24], v[25], v[26]);
  float a9 = max3(v[27], v[28], v[29]);
  float b0 = max3(a0, a1, a2), b1 = max3(a3, a4, a5), b2 = max3(a6, a7, a8), b3 = max3(a9, v[30], v[31]);
  return fmaxf(max3(b0, b1, b2), b3);
}

// Fold the maximum of one 32-column chunk into the running (max, argmax) of a row: an equal value in a later chunk never
// displaces an earlier winner, and of equal values in a chunk the lowest column wins.
// The column is found by descent: of two halves the lower one is taken when its maximum is the chunk's, and what was taken
// is halved again.  The maxima of the groups of eight fall out of the maximum itself, so a chunk costs 55 instructions where
// a key per column ((cmax - v) * 2^154 + column, reduced by minima) took 103: 100 cycles against 122 per chunk and warp with
// four warps on a scheduler, and there is no arithmetic on the values, so infinities and the largest floats are like any other.
// LAZY: the search is skipped when no row of the warp has a new maximum in this chunk - worth its branch only deep
// into a long document, where most chunks bring none.
template <bool ARGMAX, bool LAZY = false>
__device__ __forceinline__ void fold32(const float (&v)[32], int col0, float& run_m, int& run_i) {
  if (!ARGMAX) {
    run_m = fmaxf(run_m, max32(v));
    return;
  }
  float g[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) g[j] = max3(max3(v[8 * j], v[8 * j + 1], v[8 * j + 2]), max3(v[8 * j + 3], v[8 * j + 4], v[8 * j + 5]), fmaxf(v[8 * j + 6], v[8 * j + 7]));
  const float g01 = fmaxf(g[0], g[1]);
  const float cmax = max3(g01, g[2], g[3]);
  // (unconditional by default: with 32 rows per warp some row nearly always has a new maximum in a document of a few
  // chunks, and a branch costs more than the search)
  const bool better = cmax > run_m;
  if (!LAZY || __any_sync(0xffffffffu, better)) {
    float s[16], t[8], u[4];
    const bool in16 = g01 == cmax;
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = in16 ? v[i] : v[16 + i];
    const bool in8 = (in16 ? g[0] : g[2]) == cmax;
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = in8 ? s[i] : s[8 + i];
    const bool in4 = fmaxf(max3(t[0], t[1], t[2]), t[3]) == cmax;
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = in4 ? t[i] : t[4 + i];
    const bool in2 = fmaxf(u[0], u[1]) == cmax;
    const bool in1 = (in2 ? u[0] : u[2]) == cmax;
    const int p = (in16 ? 0 : 16) + (in8 ? 0 : 8) + (in4 ? 0 : 4) + (in2 ? 0 : 2) + (in1 ? 0 : 1);
    run_i = better ? col0 + p : run_i;
  }
  run_m = better ? cmax : run_m;
}
// v[i] *= scale[i]: per-column multiplier staged in shared memory
__device__ __forceinline__ void scale32(float (&v)[32], const float* scale) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const ulonglong2 sc = *reinterpret_cast<const ulonglong2*>(scale + i);
    asm("{\n\t.reg .b64 p;\n\tmov.b64 p, {%0, %1};\n\tmul.rn.f32x2 p, p, %2;\n\tmov.b64 {%0, %1}, p;\n\t}" : "+f"(v[i]), "+f"(v[i + 1]) : "l"(sc.x));
    asm("{\n\t.reg .b64 p;\n\tmov.b64 p, {%0, %1};\n\tmul.rn.f32x2 p, p, %2;\n\tmov.b64 {%0, %1}, p;\n\t}" : "+f"(v[i + 2]), "+f"(v[i + 3]) : "l"(sc.y));
  }
}
// v[i] = v[i] * scale[i] for the first `lim` columns, -inf for the others (whatever scale holds there)
__device__ __forceinline__ void scale32_first(float (&v)[32], const float* scale, int lim) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 sc = *reinterpret_cast<const float4*>(scale + i);
    v[i + 0] = i + 0 < lim ? v[i + 0] * sc.x : -INFINITY;
    v[i + 1] = i + 1 < lim ? v[i + 1] * sc.y : -INFINITY;
    v[i + 2] = i + 2 < lim ? v[i + 2] * sc.z : -INFINITY;
    v[i + 3] = i + 3 < lim ? v[i + 3] * sc.w : -INFINITY;
  }
}
// v[i] = v[i] * scale[i] + bias[i]: per-column multiplier and additive mask staged in shared memory
__device__ __forceinline__ void affine32(float (&v)[32], const float* scale, const float* bias) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 sc = *reinterpret_cast<const float4*>(scale + i);
    const float4 bi = *reinterpret_cast<const float4*>(bias + i);
    v[i + 0] = fmaf(v[i + 0], sc.x, bi.x);
    v[i + 1] = fmaf(v[i + 1], sc.y, bi.y);
    v[i + 2] = fmaf(v[i + 2], sc.z, bi.z);
    v[i + 3] = fmaf(v[i + 3], sc.w, bi.w);
  }
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                   // descriptor version for sm_100
  d |= (uint64_t)2 << 61;                   // SWIZZLE_128B
  return d;
}
// Instruction descriptor: fp32 accumulate, both operands K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t instr_desc(int ab_format, int n) {
  return (1u << 4) | ((uint32_t)ab_format << 7) | ((uint32_t)ab_format << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(TILE_M >> 4) << 24);
}

}  // namespace
}  // namespace lik
