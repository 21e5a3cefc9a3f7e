// Blackwell (sm_100a) building blocks shared by every tensor-core kernel of this
// library: mbarrier, TMA (non-multicast, tiled), tcgen05 MMA / TMEM wrappers,
// shared-memory matrix descriptors and the 128-byte swizzle helper.
//
// Every wait in this header is bounded.  A wait that runs out records where it
// gave up in a device status word and returns false; callers then leave their
// loops, fall through to the common teardown (TMEM dealloc) and return.  No
// kernel in this library traps or spins without a limit.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ctb {

// ---------------------------------------------------------------------------------------
// status word: one per device, read by the host after a step (ctb_status()).
// ---------------------------------------------------------------------------------------
struct DeviceStatus {
  unsigned int code;      // 0 = ok, otherwise first failure (kernel id << 8 | site)
  unsigned int block;     // blockIdx.x of the reporter
  unsigned int detail0;   // site specific (stage / tile / peer)
  unsigned int detail1;   // site specific (expected value / parity)
};

__device__ __forceinline__ void report_failure(DeviceStatus* st, unsigned code, unsigned d0, unsigned d1) {
  if (st == nullptr) return;
  if (atomicCAS(&st->code, 0u, code) == 0u) {
    st->block = blockIdx.x;
    st->detail0 = d0;
    st->detail1 = d1;
  }
}

// Default spin budget in clock64() ticks (~1 s at 1.9 GHz).  Tests shrink it.
#ifndef CTB_SPIN_BUDGET
#define CTB_SPIN_BUDGET (2000000000ll)
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  `abort_flag` is a shared-memory word every role of the CTA polls so
// that one role giving up ends the others quickly instead of each burning its budget.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                          DeviceStatus* st, unsigned code, long long budget = CTB_SPIN_BUDGET) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  unsigned spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 255u) == 0u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > budget) {
        *abort_flag = 1u;
        report_failure(st, code, static_cast<unsigned>(smem_u32(bar)), parity);
        return false;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// One issuing lane of a converged warp
// ---------------------------------------------------------------------------------------
// The single-thread instructions (tcgen05.mma, its commit, TMA copies) take their operands from uniform
// registers.  Inside an `if (lane == 0)` the compiler cannot keep loop-dependent operands there and moves
// them one by one: 134 cycles per MMA, whatever its shape, in a loop that chose its operands at run time,
// where a 128 x 128 x 16 product takes 65 with constant ones; four boxes of a 32 KB tile took 426 cycles to
// issue from one lane and 264 this way.  So the whole warp walks the loop with warp-uniform values and
// only the instruction itself is predicated with the lane that elect_one() chose: the *_if functions below.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t on;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b32 r;\n\t"
      "elect.sync r|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(on));
  return on;
}
// Warp index as a warp-uniform value.
__device__ __forceinline__ int uniform_warp_index() {
  return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
}
// mbar_wait by all lanes of a converged warp, which learn the same answer: lanes that left alone would be missed by the votes
// that follow, and the uniform branch is faster than the vote costs (attention, forward and backward: 1 %, a row of 1536 to 8192
// tokens backward 6 to 10 %).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                               DeviceStatus* st, unsigned code, long long budget = CTB_SPIN_BUDGET) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, st, code, budget));
}
// After a wait that gave up: the time that copies of this CTA still in flight can take at the very most (1 ms).  Their
// barriers may be among those that never completed, so there is no phase to wait for.
__device__ __forceinline__ void wait_out_copies() {
  const long long t0 = clock64();
  while (clock64() - t0 < 2000000ll) __nanosleep(1000);
}
__device__ __forceinline__ void mbar_expect_tx_if(uint32_t on, uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes), "r"(on)
      : "memory");
}

// ---------------------------------------------------------------------------------------
// proxies and fences
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(uint32_t id, uint32_t nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Barrier with an OR reduction: every one of `nthreads` threads learns whether any of
// them passed a true predicate.
__device__ __forceinline__ bool named_bar_or(uint32_t id, uint32_t nthreads, bool pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(out)
      : "r"(id), "r"(nthreads), "r"(static_cast<uint32_t>(pred))
      : "memory");
  return out != 0;
}

// ---------------------------------------------------------------------------------------
// TMA (tiled, this GPU's memory only, never cluster multicast)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_if(uint32_t on, void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x,
                                               int y) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_if(uint32_t on, void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                               int c0, int c1, int c2, int c3) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %7, 0;\n\t"
      "@q cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];\n\t}" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* smem_src, int c0, int c1, int c2,
                                             int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, const void* smem_src, int c0, int c1, int c2,
                                                  int c3) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// Untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16 bytes); the
// bytes are credited to `bar` like those of a tensor copy.
__device__ __forceinline__ void tma_load_1d_if(uint32_t on, void* smem_dst, const void* gmem_src, uint32_t bytes,
                                               uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(
          smem_u32(smem_dst)),
      "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------------------
// Programmatic dependent launch (see launch_chained in host_common.h)
// ---------------------------------------------------------------------------------------
// Every thread, before anything that the launches before this one write or read is touched; nothing to wait for in a launch
// that was not chained.
//
// A kernel that may be chained reads whatever a launch before it may have written, its weights and tables too, by ordinary loads
// through pointers that are not const __restrict__, or by load_streamed.  The read-only loads that __ldg and const __restrict__
// stand for promise that the memory does not change while the kernel runs, and this kernel runs while its predecessor still
// writes: no wait orders them, and the compiler may move them ahead of it.  (The other cache intrinsics are no better: nothing
// keeps the compiler from moving them.)  tests/test_chained_kernels.py checks the sources for it.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The launch behind this one may start when all CTAs have said so.  Not before a CTA has the TMEM that it allocates: a
// successor that took it would wait for this launch to end.
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// 16 bytes that are read once, kept behind the wait.
__device__ __forceinline__ float4 load_streamed(const float* at) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at) : "memory");
  return v;
}

// ---------------------------------------------------------------------------------------
// Cluster launch control: a CTA takes over a work item (CTA) of its grid that has not started
// ---------------------------------------------------------------------------------------
// Asks for one; the 16-byte answer is credited to `bar`.  Not to be asked again after a refusal.
__device__ __forceinline__ void work_request_if(uint32_t on, uint32_t answer, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n\t}" ::"r"(answer),
      "r"(smem_u32(bar)), "r"(on)
      : "memory");
}
// blockIdx.x of the work item taken over, -1: there is none left.
__device__ __forceinline__ int work_answer(uint32_t answer) {
  int index;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 r, [%1];\n\t"
      "mov.s32 %0, -1;\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, r;\n\t}"
      : "=r"(index)
      : "r"(answer)
      : "memory");
  return index;
}

// ---------------------------------------------------------------------------------------
// TMEM allocation (one warp, all lanes)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------------------------------
// UMMA descriptors
// ---------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, Blackwell version field = 1.
//   start address, LBO and SBO are encoded in 16-byte units.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;   // descriptor version
  d |= static_cast<uint64_t>(2) << 61;   // SWIZZLE_128B
  return d;
}
// K-major operand tile [rows][64 bf16] (128 B per row, 8-row groups 1024 B apart).
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile_addr, int k16) {
  return make_smem_desc_sw128(tile_addr + k16 * 32, 16, 1024);
}
// MN-major operand tile stored as [mn/64 atoms][k rows][64 bf16]: 8-row k groups are
// 1024 B apart (SBO), MN atoms `atom_stride` bytes apart (LBO).  One UMMA_K=16 step
// advances 16 rows = 2048 B.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile_addr, int k16, uint32_t atom_stride) {
  return make_smem_desc_sw128(tile_addr + k16 * 2048, atom_stride, 1024);
}

// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
  return (1u << 4) |                      // D format f32
         (1u << 7) |                      // A bf16
         (1u << 10) |                     // B bf16
         ((a_mn ? 1u : 0u) << 15) |       // A major
         ((b_mn ? 1u : 0u) << 16) |       // B major
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// D += A B for the lane with `on` set (see elect_one); both operands in shared memory.
__device__ __forceinline__ void umma_bf16_if(uint32_t on, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// A operand from TMEM (bf16 packed two per 32-bit column), B from shared memory.
__device__ __forceinline__ void umma_bf16_ts_if(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b,
                                                uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// Arrive on an mbarrier once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit_if(uint32_t on, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
      "r"(on)
      : "memory");
}

// ---------------------------------------------------------------------------------------
// TMEM loads: 32 lanes x 32-bit, N consecutive columns into N registers per thread.
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
// 128 consecutive columns of this thread's lane: four loads in flight, one wait by the caller.
__device__ __forceinline__ void tmem_ld32x4(uint32_t taddr, uint32_t (&r)[128]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld32(taddr + c * 32, reinterpret_cast<uint32_t(&)[32]>(r[c * 32]));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------------------
// 128-byte swizzle: byte offset of 16-byte chunk `chunk` (0..7) of row `row` inside a
// tile whose rows are 128 B and whose base is 1024-byte aligned.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed fp32 pairs (sm_100 f32x2 arithmetic: one instruction for two lanes of the FMA pipe).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// exp2 of a packed pair on the FMA pipe, for a share of the exponentials of kernels whose ex2 unit (16 a
// clock per SM) is the busiest pipe.  x = n + f with n = round(x) by the 1.5 * 2^23 addition, 2^f on
// [-1/2, 1/2] by the degree-5 minimax polynomial of the relative error (Remez; 7.7e-8, 2.1e-7 with the
// rounding of its fp32 steps, where ex2.approx allows 2.4e-7), times 2^n built in the exponent field.
// Arguments below -125 count as -125 (no zero result), above 127 are not meant; NaN stays NaN.
__device__ __forceinline__ void poly_exp2_x2(uint64_t x2, float& ya, float& yb) {
  const uint64_t magic = pack_f32x2(12582912.f, 12582912.f), minus = pack_f32x2(-1.f, -1.f);
  float xa, xb, ta, tb;
  unpack_f32x2(x2, xa, xb);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(xa) : "f"(-125.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(xb) : "f"(-125.f));
  x2 = pack_f32x2(xa, xb);
  const uint64_t t2 = add_f32x2(x2, magic);
  const uint64_t f2 = add_f32x2(x2, fma_f32x2(t2, minus, magic));
  uint64_t p2 = fma_f32x2(pack_f32x2(0.0013277939287945628f, 0.0013277939287945628f), f2,
                          pack_f32x2(0.009675757959485054f, 0.009675757959485054f));
  p2 = fma_f32x2(p2, f2, pack_f32x2(0.05550709739327431f, 0.05550709739327431f));
  p2 = fma_f32x2(p2, f2, pack_f32x2(0.24022114276885986f, 0.24022114276885986f));
  p2 = fma_f32x2(p2, f2, pack_f32x2(0.6931469440460205f, 0.6931469440460205f));
  p2 = fma_f32x2(p2, f2, pack_f32x2(1.0000001192092896f, 1.0000001192092896f));
  unpack_f32x2(t2, ta, tb);
  const uint64_t n2 = pack_f32x2(__uint_as_float((__float_as_uint(ta) << 23) + 0x3f800000u),
                                 __uint_as_float((__float_as_uint(tb) << 23) + 0x3f800000u));
  unpack_f32x2(mul_f32x2(p2, n2), ya, yb);
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Bit masks over positions 0..31: positions >= x, positions <= x (x may lie outside 0..31).
__device__ __forceinline__ unsigned bits_from(int x) { return x <= 0 ? 0xffffffffu : (x >= 32 ? 0u : 0xffffffffu << x); }
__device__ __forceinline__ unsigned bits_upto(int x) { return x < 0 ? 0u : (x >= 31 ? 0xffffffffu : 0xffffffffu >> (31 - x)); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

}  // namespace ctb
