// sm_100a PTX wrappers used by the attention-forward kernels: mbarrier (bounded waits),
// TMA tiled loads/stores, tcgen05 (TMEM alloc, MMA, commit, ld/st, fences), setmaxnreg.
//
// These replace the reference's sm_120 helper set (include/utils.h:25-140 of the reference:
// mma.sync m16n8k16, ldmatrix, unbounded mbarrier spin, 3-D TMA without swizzle).
// Nothing here is shared with that file: the tensor path is tcgen05 + TMEM, every wait
// has an iteration limit, and TMA uses 128-byte swizzle so that the same shared-memory
// image is directly consumable by a UMMA shared-memory descriptor.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_fp16.h>

namespace fa {

// ---------------------------------------------------------------------------------------
// generic helpers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "elect.sync _|P, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

template <uint32_t N>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N));
}
template <uint32_t N>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N));
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// sm_100 three-input max and two-wide fp32 arithmetic (one issue slot for two lanes of work)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// 0xFFFF in each half where a < b as fp16
__device__ __forceinline__ uint32_t f16x2_less_mask(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("set.lt.u32.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// the larger of two values, NaN if either is
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// two floats -> packed fp16x2, round-to-nearest-even; `lo` lands in bits [15:0]
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Programmatic dependent launch: a grid launched with that attribute may start before the grid in front of it in the
// stream has ended. griddep_wait() holds a thread until that grid has completed and its memory is visible;
// griddep_launch() (once per CTA) lets the grid behind this one start where SMs are free. Both do nothing in a grid
// that was launched without the attribute or has no such successor.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// generic-proxy writes to shared memory -> visible to the async proxy (TMA, UMMA operand reads)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrival by lane 0 of a warp, without a branch.
__device__ __forceinline__ void mbar_arrive_lane0(uint64_t* bar, int lane) {
  asm volatile("{\n.reg .pred p;\nsetp.eq.s32 p, %1, 0;\n@p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(smem_u32(bar)), "r"(lane) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.u32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. Returns true when the phase completed, false when the limit ran out or another role already
// gave up (`*abort_flag != 0`). A probe of a phase that has not completed suspends the thread in hardware for
// about 4 us (7.8 k SM cycles, measured on B200) or until the phase completes, whichever comes first, so the limit
// is a number of probes: 2^18 of them are about one second. A protocol bug therefore turns into a status word on
// the host instead of a hung GPU.
#ifndef FA_WAIT_LIMIT_POLLS
#define FA_WAIT_LIMIT_POLLS (1u << 18)
#endif

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  // Between two probes stand a counter and its test; the abort flag is read after every 64th only: what sits there is
  // added to every hand-off in the kernels (a loop that read the flag after each probe cost 5 % of the whole attention
  // kernel). Written as one block of PTX, a wait is 11 instructions in each of its
  // many places; as C++ around single probes it came to 40, 27 KB of the kernel, and the first and last rounds of an
  // item, whose code is rarely in the instruction caches, ran slower: B4 H16 N2048 d64 causal 72.0 -> 67.8 us, B8 H12
  // N1000 d64 54.5 -> 51.6, B8 H16 N1024 d128 61.5 -> 58.2.
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred P, Q;\n"
      ".reg .u32 n, f;\n"
      "mov.u32 n, 0;\n"
      "PROBE:\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "@P bra DONE;\n"
      "add.u32 n, n, 1;\n"
      "and.b32 f, n, 63;\n"
      "setp.ne.u32 Q, f, 0;\n"
      "@Q bra PROBE;\n"
      "ld.volatile.shared.u32 f, [%3];\n"
      "setp.ne.u32 Q, f, 0;\n"
      "@Q bra DONE;\n"
      "setp.lt.u32 Q, n, %4;\n"
      "@Q bra PROBE;\n"
      "st.volatile.shared.u32 [%3], 1;\n"
      "DONE:\n"
      "selp.u32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(smem_u32(const_cast<int*>(abort_flag))), "n"(FA_WAIT_LIMIT_POLLS)
      : "memory");
  return ok != 0;
}

// Same, for a whole warp polling one barrier: the verdict is made warp-uniform so that a
// give-up never splits a warp in front of a .sync.aligned instruction.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// ---------------------------------------------------------------------------------------
// TMA (tiled, 4-D maps: {64 contiguous fp16, row, 64-wide panel, head})
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// Loads one box into shared memory and completes `bytes` on the mbarrier. c0 must keep
// c0 * 2 bytes a multiple of 16 (it is always 0 here).
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
      : "memory");
}

// Stores one box from shared memory (same swizzled layout as a load) as a bulk group of the issuing thread; rows of
// the box beyond the tensor's extent are not written. c0 * 2 bytes must be a multiple of 16 (it is always 0 here) and
// no coordinate may be negative.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* smem_src, int c0, int c1, int c2,
                                             int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group"
      " [%0, {%2, %3, %4, %5}], [%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// The issuing thread's bulk stores have finished reading shared memory (the source may be overwritten).
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// The issuing thread's bulk stores are complete.
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------------------------------
// tcgen05: tensor memory management
// ---------------------------------------------------------------------------------------
// Warp-wide. Writes the TMEM base address (lane 0, first column) into *smem_slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// TMEM address = (lane << 16) | column. A warp may touch only lanes 32*(warp%4) .. +31.
__device__ __forceinline__ uint32_t tmem_addr(uint32_t base, uint32_t lane, uint32_t col) {
  return base + (lane << 16) + col;
}

// ---------------------------------------------------------------------------------------
// tcgen05: MMA
// ---------------------------------------------------------------------------------------
// Instruction descriptor for kind::f16 with fp16 A/B and fp32 accumulator.
//   [4,6)  D format (1 = f32)     [7,10) A format (0 = f16)   [10,13) B format (0 = f16)
//   [15]   A major (0 = K)        [16]   B major (0 = K, 1 = MN)
//   [17,23) N >> 3                [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc_f16(uint32_t M, uint32_t N, uint32_t a_mn_major,
                                                      uint32_t b_mn_major) {
  return (1u << 4) | (0u << 7) | (0u << 10) | (a_mn_major << 15) | (b_mn_major << 16) | ((N >> 3) << 17) |
         ((M >> 4) << 24);
}

// Shared-memory matrix descriptor, 128-byte swizzle.
//   [0,14) start >> 4   [16,30) leading-dim byte offset >> 4   [32,46) stride-dim byte offset >> 4
//   [46,48) descriptor version (1 on sm_100)   [61,64) layout (2 = SWIZZLE_128B)
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Groups of products issued by a converged warp: one elected lane issues them under a guard predicate, in one block
// without branches. The 32 products and six satisfied waits of a round at head_dim 128, issued in a loop of their own
// beside eight softmax warps: 2985 clocks as `if (elect_one()) { products } __syncwarp();` with a vote behind each wait,
// 2547 in this form, 2366 in this form without the votes; 24 products at head_dim 64 2482, 2093, 1934.
// Descriptors are given as their low words (start address and leading-dimension offset); the high words are a constant.
// D (+)= P V for 64 keys: P at `p_tmem`, 8 columns per product; V read MN-major, 2048 bytes per product.
__device__ __forceinline__ void umma_pv64(uint32_t d_tmem, uint32_t p_tmem, uint32_t v_lo, uint32_t hi, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred lead, acc, yes;\n"
      ".reg .b64 v;\n"
      ".reg .b32 lo, p;\n"
      "elect.sync _|lead, 0xffffffff;\n"
      "setp.ne.b32 acc, %5, 0;\n"
      "setp.eq.b32 yes, 0, 0;\n"
      "mov.b64 v, {%2, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], v, %4, acc;\n"
      "add.u32 lo, %2, 128;\n add.u32 p, %1, 8;\n mov.b64 v, {lo, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [p], v, %4, yes;\n"
      "add.u32 lo, %2, 256;\n add.u32 p, %1, 16;\n mov.b64 v, {lo, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [p], v, %4, yes;\n"
      "add.u32 lo, %2, 384;\n add.u32 p, %1, 24;\n mov.b64 v, {lo, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [p], v, %4, yes;\n"
      "}\n"
      :
      : "r"(d_tmem), "r"(p_tmem), "r"(v_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D += P V for 32 keys.
__device__ __forceinline__ void umma_pv32(uint32_t d_tmem, uint32_t p_tmem, uint32_t v_lo, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n"
      ".reg .pred lead, yes;\n"
      ".reg .b64 v;\n"
      ".reg .b32 lo, p;\n"
      "elect.sync _|lead, 0xffffffff;\n"
      "setp.eq.b32 yes, 0, 0;\n"
      "mov.b64 v, {%2, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], v, %4, yes;\n"
      "add.u32 lo, %2, 128;\n add.u32 p, %1, 8;\n mov.b64 v, {lo, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], [p], v, %4, yes;\n"
      "}\n"
      :
      : "r"(d_tmem), "r"(p_tmem), "r"(v_lo), "r"(hi), "r"(idesc)
      : "memory");
}
// D (+)= P V for 96 keys.
__device__ __forceinline__ void umma_pv96(uint32_t d_tmem, uint32_t p_tmem, uint32_t v_lo, uint32_t hi, uint32_t idesc,
                                          uint32_t accumulate) {
  umma_pv64(d_tmem, p_tmem, v_lo, hi, idesc, accumulate);
  umma_pv32(d_tmem, p_tmem + 32, v_lo + 512, hi, idesc);
}
// D (+)= Q K^T over 64 elements of head_dim (one 128-byte panel), 32 bytes per product.
__device__ __forceinline__ void umma_qk64(uint32_t d_tmem, uint32_t q_lo, uint32_t k_lo, uint32_t hi, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred lead, acc, yes;\n"
      ".reg .b64 q, k;\n"
      ".reg .b32 a, b;\n"
      "elect.sync _|lead, 0xffffffff;\n"
      "setp.ne.b32 acc, %5, 0;\n"
      "setp.eq.b32 yes, 0, 0;\n"
      "mov.b64 q, {%1, %3};\n mov.b64 k, {%2, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], q, k, %4, acc;\n"
      "add.u32 a, %1, 2;\n add.u32 b, %2, 2;\n mov.b64 q, {a, %3};\n mov.b64 k, {b, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], q, k, %4, yes;\n"
      "add.u32 a, %1, 4;\n add.u32 b, %2, 4;\n mov.b64 q, {a, %3};\n mov.b64 k, {b, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], q, k, %4, yes;\n"
      "add.u32 a, %1, 6;\n add.u32 b, %2, 6;\n mov.b64 q, {a, %3};\n mov.b64 k, {b, %3};\n"
      "@lead tcgen05.mma.cta_group::1.kind::f16 [%0], q, k, %4, yes;\n"
      "}\n"
      :
      : "r"(d_tmem), "r"(q_lo), "r"(k_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// umma_commit() by one elected lane of a converged warp, if `cond`.
__device__ __forceinline__ void umma_commit_warp(uint64_t* bar, bool cond = true) {
  asm volatile(
      "{\n"
      ".reg .pred lead, c;\n"
      "elect.sync _|lead, 0xffffffff;\n"
      "setp.ne.and.b32 c, %1, 0, lead;\n"
      "@c tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(smem_u32(bar)), "r"(static_cast<uint32_t>(cond))
      : "memory");
}
// The mbarrier receives one arrival when every tcgen05 operation issued so far by this
// thread has completed. Implies tcgen05.fence::before_thread_sync.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ---------------------------------------------------------------------------------------
// tcgen05: TMEM <-> registers, shape 32x32b (thread i of the warp <-> lane base+i,
// register j <-> column base+j)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]),
        "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// tcgen05.ld writes its destination registers asynchronously; tcgen05.wait::ld makes them valid.
// Nothing ties the registers to the wait instruction in the compiler's eyes, so after the wait
// each loaded array is passed through this empty statement: it keeps every later use of the
// registers behind the wait without emitting an instruction.
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[32]) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

__device__ __forceinline__ void tmem_ld_fence16(uint32_t (&r)[16]) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15])
               :
               : "memory");
}

__device__ __forceinline__ void tmem_ld_fence8(uint32_t (&r)[8]) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld_fence_cols(uint32_t (&r)[8]) { tmem_ld_fence8(r); }
__device__ __forceinline__ void tmem_ld_fence_cols(uint32_t (&r)[16]) { tmem_ld_fence16(r); }

// ---------------------------------------------------------------------------------------
// CTA pairs (cluster of 2): cta_group::2 MMA, multicast commit, remote mbarrier arrival
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local_smem_addr` in the CTA of rank `rank`
__device__ __forceinline__ uint32_t mapa_u32(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
  return r;
}
// Arrival on an mbarrier of any CTA of the cluster (address from mapa_u32), with the default (CTA-scope
// release) ordering. A cluster-scope release (.release.cluster) stalls the arriving warp for a fence of
// several hundred cycles, which cost a third of the pair kernel's throughput; it is not needed where what
// the arrival announces is not generic-proxy memory of the arriving thread: tensor-memory contents
// (ordered by tcgen05.wait + tcgen05.fence::before_thread_sync), or a TMA write into this CTA's shared
// memory that this CTA's own tensor core will read.
__device__ __forceinline__ void mbar_arrive_peer(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// One instruction for both CTAs of the pair (issued by one thread of the even-ranked CTA): M = 256
// rows (128 per CTA, each from its own shared memory / TMEM at the same offsets), B split along N
// (CTA r supplies columns [r*N/2, (r+1)*N/2) from its own shared memory), D rows land in each CTA's TMEM.
__device__ __forceinline__ void umma_ss_2cta(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_ts_2cta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the mbarrier at this shared-memory offset in every CTA of `cta_mask` once all
// tcgen05 operations issued so far by this thread have completed
__device__ __forceinline__ void umma_commit_2cta(uint64_t* bar, uint16_t cta_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(cta_mask)
      : "memory");
}

}  // namespace fa
