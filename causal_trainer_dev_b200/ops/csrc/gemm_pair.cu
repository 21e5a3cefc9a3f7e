// Two-CTA tcgen05 GEMM: a cluster of two CTAs on two SMs computes one 256 x 256 (or 512 x 256) output tile with
// `tcgen05.mma.cta_group::2`.  Each CTA stages its own 128 rows of A and its own 128 columns of B, and the
// tensor cores of both SMs read both halves of B.
//
//   C[M,N] = alpha * A * B^T   and the epilogues of gemm_epilogue.cuh, the four operand layouts of gemm.cu
//
// What it is for.  An SM takes at most 64 bytes a clock from L2.  A k-block of a one-CTA 128 x 256 tile is
// 48 KB for 516 cycles of tensor core, so that tile runs at two thirds of the tensor rate at best (1000 x 17920 x 1536, counters:
// 661 MB from L2, 61 bytes a clock and SM while it works, the tensor pipe active for 65 % of it).  Here a k-block is 32 KB for the
// same 516 cycles (440 MB, 75 %).  Long products run under the power cap, where bytes cost clock: the taller tile reads less
// of B, and bands of 16 row tiles re-read B from memory half as often.  One-CTA kernels and here, the two in turn for 4 s in
// blocks of 20 ms, medians in us with the tenth and ninetieth hundredths: 16384 x 28672 x 4096 3090 (2972..3176) and 2768
// (2686..2877), 16384 x 14336 x 4096 of a gradient 1533 (1499..1606) and 1390 (1365..1447), 4096 x 14336 x 16384 1587 (1517..1624) and
// 1398 (1313..1441), 28672 x 4096 x 16384 3088 (2953..3219) and 2902 (2789..3222), 4096 x 4096 x 128256 4306 (4233..4424) and 3293
// (3247..3401), 8192 x 1536 x 17920 412 (404..425) and 349 (343..358), 8192 x 17920 x 1536 423 (385..453) and 340 (323..382), 1000 x 17920 x
// 1536 58 (57..59) and 51 (51..52).  16384 x 4096 x 14336 and x 28672 stay on one CTA.  Of that little is left in a whole pass over
// an 8B MLP, whose products warm the chip for one another: 14.20 ms before there was this choice, 14.09 with it.
//
// Tiles of a wave that would be nearly empty, or all of them where they are fewer than the pairs of SMs, may be cut
// along K into slices that leave fp32 partial tiles in a workspace; a second kernel adds them in the order of the slices, so
// the result does not depend on timing.
//
// Roles per CTA: warp 0 TMA producer (each CTA loads its own operands; the bytes of both are credited to the full
// barrier of the leader CTA), warp 1 of the leader issues the MMAs for the pair and releases stages / publishes
// accumulators with multicast commits to both CTAs, warp 2 owns the TMEM allocation, warps 4-11 drain this CTA's
// accumulator rows.  256 x 256 tiles double-buffer the accumulator in the two 256-column TMEM slots.  Every wait is
// bounded; the two CTAs meet at a cluster barrier before they tear down, so neither leaves while the other can still
// signal it.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "gemm_epilogue.cuh"

namespace ctb {
namespace gemm2 {

using gemm::BM;
using gemm::BN;
using gemm::EPI_BUF;
constexpr int BK = 64;
constexpr int BNH = 128;                 // columns of B staged per CTA
constexpr int B_STAGE = BNH * BK * 2;    // 16 KiB

// A pair's tile is TM sub-tiles of 256 rows that share B.  Two epilogue warpgroups: with TM = 2 each drains the slot of
// one sub-tile, with TM = 1 each drains half of the columns (the loss statistics, which want whole slabs, take one).
template <int TM, int EPI>
struct Cfg {
  static constexpr int NSTAGE = TM == 1 ? 6 : 4;
  static constexpr int A_STAGE = TM * BM * BK * 2;
  static constexpr int OFF_B = NSTAGE * A_STAGE;
  static constexpr int OFF_EPI = OFF_B + NSTAGE * B_STAGE;
  static constexpr int OFF_BAR = OFF_EPI + 2 * EPI_BUF;
  static constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
  static constexpr int EPI_GROUPS = (TM == 1 && EPI == EPI_CE_STATS) ? 1 : 2;
  static constexpr int EPI_COLS = TM == 1 ? BN / EPI_GROUPS : BN;      // columns that a warpgroup drains
  static constexpr int EPI_BUFS = 2 / EPI_GROUPS;
  static constexpr int THREADS = 128 + 128 * EPI_GROUPS;
};

enum : unsigned {
  SITE_P_EMPTY = 0x0801,
  SITE_P_FULL = 0x0802,
  SITE_P_TEMPTY = 0x0803,
  SITE_P_TFULL = 0x0804,
};

// Work units: whole tiles [0, whole), then `slices` K slices of each of the tiles behind them, whose fp32
// partial tiles go to the workspace.
struct PairArgs {
  int num_m, num_n, num_k;
  int whole, slices, units;
  int band;                // row tiles per band of the tile walk
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory object in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Tensor copy into this CTA's shared memory whose bytes are credited to a barrier of the pair
// (`bar_cluster_addr` is a shared::cluster address, here always the leader's).
__device__ __forceinline__ void tma_load_2d_pair_if(uint32_t on, void* smem_dst, const CUtensorMap* map,
                                                    uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_pair_if(uint32_t on, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                                  uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once all MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair_if(uint32_t on, uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(
          smem_u32(bar)),
      "h"(mask), "r"(on)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

struct Unit {
  int m0, n0;        // first row and column of the pair's tile
  int kb0, kb1;      // its k-blocks
  int part;          // index of the partial tile in the workspace, -1 for a whole tile
};
// Bands of `band` row tiles; inside a band the column advances slowly (B stays hot in L2).
template <int TM>
__device__ __forceinline__ Unit map_unit(int unit, const PairArgs& p) {
  Unit u;
  int tile = unit;
  u.kb0 = 0;
  u.kb1 = p.num_k;
  u.part = -1;
  if (unit >= p.whole) {
    // neighbours work on the same slice of different tiles: they share its operands in L2
    const int rest = p.num_m * p.num_n - p.whole;
    u.part = unit - p.whole;
    const int slice = u.part / rest;
    tile = p.whole + u.part - slice * rest;
    u.kb0 = static_cast<int>(static_cast<long>(p.num_k) * slice / p.slices);
    u.kb1 = static_cast<int>(static_cast<long>(p.num_k) * (slice + 1) / p.slices);
  }
  const int per_band = p.band * p.num_n;
  const int first_m = tile / per_band * p.band;
  const int rows = min(p.band, p.num_m - first_m);
  const int local = tile % per_band;
  u.m0 = (first_m + local % rows) * 2 * TM * BM;
  u.n0 = (local / rows) * BN;
  return u;
}

template <int TM, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(512, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_part,
                 const GemmArgs args, const PairArgs walk) {
  using C = Cfg<TM, EPI>;
  constexpr int NSTAGE = C::NSTAGE;
  constexpr int A_STAGE = C::A_STAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);   // used in the leader only
  uint64_t* empty = full + NSTAGE;
  uint64_t* tfull = empty + NSTAGE;      // [2]
  uint64_t* tempty = tfull + 2;          // [2] used in the leader only: both CTAs' epilogue warps arrive
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  DeviceStatus* st = args.status;
  const long long budget = args.spin_budget;
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], TM == 1 ? 8 * C::EPI_GROUPS : 8);      // the epilogue warps of both CTAs
    }
    *abort_flag = 0u;
    mbar_fence_init();
  }
  if (warp == 3 && lane == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    if (EPI != EPI_CE_STATS) tma_prefetch_desc(&map_c);
  }
  if (warp == 2) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                    // both CTAs' barriers exist before either signals the other
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (args.chained) let_successor_start();
  wait_for_predecessor();

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    const uint32_t on = elect_one();             // the whole warp walks, one lane issues
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int unit = pair; ok && unit < walk.units; unit += pairs) {
      const Unit u = map_unit<TM>(unit, walk);
      const int m0 = u.m0 + static_cast<int>(rank) * BM;       // this CTA's rows of A (of every 256-row sub-tile)
      const int n0 = u.n0 + static_cast<int>(rank) * BNH;      // this CTA's columns of B
      for (int kb = u.kb0; kb < u.kb1; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag, st, SITE_P_EMPTY, budget)) {
          ok = false;
          break;
        }
        // the leader arms its barrier with the bytes of both CTAs
        if (leader) mbar_expect_tx_if(on, &full[stage], 2 * (A_STAGE + B_STAGE));
        const uint32_t bar = map_to_rank(smem_u32(&full[stage]), 0);
        uint8_t* sa = smem + stage * A_STAGE;
        uint8_t* sb = smem + C::OFF_B + stage * B_STAGE;
        const int k0 = kb * BK;
#pragma unroll
        for (int h = 0; h < TM; ++h) {
          if (A_MN) {
#pragma unroll
            for (int a = 0; a < BM / 64; ++a)
              tma_load_2d_pair_if(on, sa + h * 16384 + a * 8192, &map_a, bar, m0 + h * 2 * BM + a * 64, k0);
          } else {
            tma_load_2d_pair_if(on, sa + h * 16384, &map_a, bar, k0, m0 + h * 2 * BM);
          }
        }
        if (B_MN) {
#pragma unroll
          for (int a = 0; a < BNH / 64; ++a) tma_load_2d_pair_if(on, sb + a * 8192, &map_b, bar, n0 + a * 64, k0);
        } else {
          tma_load_2d_pair_if(on, sb, &map_b, bar, k0, n0);
        }
        if (++stage == NSTAGE) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok || *abort_flag) {
      // leave no copy of this CTA in flight: they are credited to the leader's barriers, which the peer may no longer
      // arm, so wait out the time that local copies can take at the very most (1 ms) instead of a phase
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) __nanosleep(1000);
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA, for the pair) ------------------------------
    if (leader) {
      const uint32_t on = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      uint32_t stage = 0, phase = 0;
      uint32_t uses0 = 0, uses1 = 0;       // completed uses of the two TMEM slots
      uint32_t next_slot = 0;              // TM == 1: slots alternate from tile to tile
      bool ok = true;
      for (int unit = pair; ok && unit < walk.units; unit += pairs) {
        const Unit u = map_unit<TM>(unit, walk);
        // the slots must have been drained by both CTAs' epilogues of the tile that used them last
        if (TM == 2 || next_slot == 0)
          ok = mbar_wait_warp(&tempty[0], (uses0 & 1u) ^ 1u, abort_flag, st, SITE_P_TEMPTY, budget);
        if (ok && (TM == 2 || next_slot == 1))
          ok = mbar_wait_warp(&tempty[1], (uses1 & 1u) ^ 1u, abort_flag, st, SITE_P_TEMPTY, budget);
        if (!ok) break;
        tc_fence_after();
        for (int kb = u.kb0; kb < u.kb1; ++kb) {
          if (!mbar_wait_warp(&full[stage], phase, abort_flag, st, SITE_P_FULL, budget)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * A_STAGE);
          const uint32_t sb = smem_u32(smem + C::OFF_B + stage * B_STAGE);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t db = B_MN ? desc_mnmajor(sb, k, 8192) : desc_kmajor(sb, k);
#pragma unroll
            for (int h = 0; h < TM; ++h) {
              const uint64_t da = A_MN ? desc_mnmajor(sa + h * 16384, k, 8192) : desc_kmajor(sa + h * 16384, k);
              umma_bf16_pair_if(on, tmem_base + (TM == 1 ? next_slot : h) * BN, da, db, idesc,
                                (kb != u.kb0 || k != 0) ? 1u : 0u);
            }
          }
          umma_commit_pair_if(on, &empty[stage]);       // both producers may refill the stage
          if (++stage == NSTAGE) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        // both epilogues may drain the slots
        if (TM == 2 || next_slot == 0) {
          umma_commit_pair_if(on, &tfull[0]);
          ++uses0;
        }
        if (TM == 2 || next_slot == 1) {
          umma_commit_pair_if(on, &tfull[1]);
          ++uses1;
        }
        next_slot ^= 1u;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------ epilogue: this CTA's 128 accumulator rows ------------------------------
    const int wg = (warp - 4) >> 2;
    const int slot_of = TM == 1 ? 0 : wg;                     // sub-tile and first column of this warpgroup
    const int col_of = TM == 1 ? wg * C::EPI_COLS : 0;
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int etid = threadIdx.x - 128 - wg * 128;
    const uint32_t bar_stage = 1 + wg, bar_vote = 3 + wg;
    uint32_t used = 0;                       // bit s: parity of the uses of slot s
    uint32_t next_slot = 0, staged = 0;
    uint8_t* epi = smem + C::OFF_EPI + wg * EPI_BUF;
    for (int unit = pair; unit < walk.units; unit += pairs) {
      const Unit u = map_unit<TM>(unit, walk);
      const uint32_t slot = TM == 1 ? next_slot : static_cast<uint32_t>(slot_of);
      const bool ready = mbar_wait(&tfull[slot], (used >> slot) & 1u, abort_flag, st, SITE_P_TFULL, budget);
      if (named_bar_or(bar_vote, 128, !ready)) break;      // the four warps decide together
      used ^= 1u << slot;
      next_slot ^= 1u;
      tc_fence_after();
      const uint32_t taddr = tmem_base + slot * BN + col_of + (static_cast<uint32_t>(q * 32) << 16);
      const int m_sub = u.m0 + slot_of * 2 * BM + static_cast<int>(rank) * BM;
      if (EPI == EPI_STORE && u.part >= 0) {
        // fp32 partial tile [256 TM][256] of the workspace
        const int y = (u.part * 2 * TM + slot_of * 2 + static_cast<int>(rank)) * BM + q * 32;
        gemm::drain_f32<C::EPI_COLS, C::EPI_BUFS>(taddr, 1.f, C::EPI_COLS, epi + q * 4096, staged, lane, &map_part, col_of, y,
                                                  false);
      } else {
        gemm::drain_slot<EPI, C::EPI_COLS, C::EPI_BUFS>(args, &map_c, taddr, u.n0 + col_of, m_sub, row, etid, bar_stage, epi,
                                                        staged, args.accumulate != 0);
      }
      tc_fence_before();
      __syncwarp();
      // the leader's MMA warp counts the epilogue warps of the pair
      if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&tempty[slot]), 0));
    }
    if (lane == 0) tma_wait_group<0>();
  }

  // ------------------------------ teardown ------------------------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync();                    // nobody leaves while its peer may still signal it
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Sum of the partial tiles in slice order, a warp per row of a tile, eight columns a thread.
template <int TM, bool F32>
__global__ void __launch_bounds__(256) pair_reduce_kernel(const float* part, const GemmArgs args, const PairArgs walk,
                                                          void* out, long ldc) {
  if (args.chained) let_successor_start();
  wait_for_predecessor();
  constexpr int ROWS = 2 * TM * BM;
  const int rest = walk.num_m * walk.num_n - walk.whole;
  const int tile = blockIdx.x / (ROWS / 8);
  const int row = (blockIdx.x % (ROWS / 8)) * 8 + (threadIdx.x >> 5);
  const int col = (threadIdx.x & 31) * 8;
  const Unit u = map_unit<TM>(walk.whole + tile, walk);
  const int m = u.m0 + row, n = u.n0 + col;
  if (m >= args.M || n >= args.N) return;
  const float* from = part + (static_cast<size_t>(tile) * ROWS + row) * BN + col;
  const size_t step = static_cast<size_t>(rest) * ROWS * BN;
  float4 lo = load_streamed(from), hi = load_streamed(from + 4);
  for (int s = 1; s < walk.slices; ++s) {
    const float4 a = load_streamed(from + s * step), b = load_streamed(from + s * step + 4);
    lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
    hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
  }
  float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (!F32 && args.bias != nullptr && n + e < args.N) v[e] += __bfloat162float(args.bias[n + e]);
    v[e] *= args.alpha;
  }
  const size_t to = static_cast<size_t>(m) * ldc + n;
  if (F32) {
    float* dst = static_cast<float*>(out) + to;
    if (n + 8 <= args.N) {
      reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (n + e < args.N) dst[e] = v[e];
    }
  } else {
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(out) + to;
    if (n + 8 <= args.N) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                                                  pack_bf16(v[6], v[7]));
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (n + e < args.N) dst[e] = __float2bfloat16(v[e]);
    }
  }
}

template <int TM, bool A_MN, bool B_MN, int EPI>
int launch(const TensorMap& ma, const TensorMap& mb, const TensorMap& mc, const TensorMap& mp, const GemmArgs& a,
           const PairArgs& w, cudaStream_t s) {
  auto kern = gemm_pair_kernel<TM, A_MN, B_MN, EPI>;
  static int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    CTB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<TM, EPI>::SMEM_BYTES));
    configured_dev = dev;
  }
  CTB_CUDA_OK(launch_chained(a.chained != 0, kern, 2 * std::min(w.units, sm_count() / 2), Cfg<TM, EPI>::THREADS,
                             Cfg<TM, EPI>::SMEM_BYTES, s, 2, ma.map, mb.map, mc.map, mp.map, a, w));
  return 0;
}

template <int TM, int EPI>
int dispatch(const GemmCall& c, const TensorMap& ma, const TensorMap& mb, const TensorMap& mc, const TensorMap& mp,
             const GemmArgs& a, const PairArgs& w) {
  cudaStream_t s = static_cast<cudaStream_t>(c.stream);
  if (!c.a_mn && !c.b_mn) return launch<TM, false, false, EPI>(ma, mb, mc, mp, a, w, s);
  if (EPI != EPI_STORE) return fail("gemm: the loss epilogues take K-major operands");
  if (!c.a_mn && c.b_mn) return launch<TM, false, true, EPI_STORE>(ma, mb, mc, mp, a, w, s);
  if (c.a_mn && c.b_mn) return launch<TM, true, true, EPI_STORE>(ma, mb, mc, mp, a, w, s);
  return launch<TM, true, false, EPI_STORE>(ma, mb, mc, mp, a, w, s);
}

template <int TM>
int run(const GemmCall& c, const PairPlan& plan) {
  const TensorMap ma = c.a_mn ? get_tensor_map_2d(c.A, Elt::BF16, c.M, c.K, c.lda, 64, 64, true)
                             : get_tensor_map_2d(c.A, Elt::BF16, c.K, c.M, c.lda, 64, 128, true);
  const TensorMap mb = c.b_mn ? get_tensor_map_2d(c.B, Elt::BF16, c.N, c.K, c.ldb, 64, 64, true)
                             : get_tensor_map_2d(c.B, Elt::BF16, c.K, c.N, c.ldb, 64, 128, true);
  if (!ma || !mb) return 1;
  GemmArgs a{};
  a.chained = chained_call(c);
  a.M = c.M;
  a.N = c.N;
  a.K = c.K;
  a.out_f32 = c.out_f32;
  a.accumulate = c.accumulate;
  a.alpha = c.alpha;
  a.bias = static_cast<const __nv_bfloat16*>(c.bias);
  a.status = device_status();
  a.spin_budget = c.spin_budget > 0 ? c.spin_budget : CTB_SPIN_BUDGET;
  a.ce_targets = c.ce_targets;
  a.ce_target_step = c.ce_target_step;
  a.ce_max = c.ce_max;
  a.ce_sum = c.ce_sum;
  a.ce_target_logit = c.ce_target_logit;
  a.ce_lse = c.ce_lse;
  a.ce_coef = c.ce_coef;
  a.ce_keep = c.epi == EPI_CE_STATS && c.C != nullptr;
  PairArgs w{};
  w.num_m = (c.M + 2 * TM * BM - 1) / (2 * TM * BM);
  w.num_n = (c.N + BN - 1) / BN;
  w.num_k = (c.K + BK - 1) / BK;
  w.whole = plan.whole;
  w.slices = plan.slices;
  w.band = plan.band;
  const int rest = w.num_m * w.num_n - w.whole;
  w.units = w.whole + rest * w.slices;
  TensorMap mc = ma;      // placeholder where no C tensor is written
  if (c.epi != EPI_CE_STATS || c.C != nullptr) {
    mc = c.out_f32 ? get_tensor_map_2d(c.C, Elt::F32, c.N, c.M, c.ldc, 32, 32, true)
                   : get_tensor_map_2d(c.C, Elt::BF16, c.N, c.M, c.ldc, 64, 32, true);
    if (!mc) return 1;
  }
  TensorMap mp = ma;
  if (rest > 0) {
    mp = get_tensor_map_2d(c.workspace, Elt::F32, BN, static_cast<uint64_t>(rest) * w.slices * 2 * TM * BM, BN, 32, 32, true);
    if (!mp) return 1;
  }
  int rc = 0;
  switch (c.epi) {
    case EPI_STORE: rc = dispatch<TM, EPI_STORE>(c, ma, mb, mc, mp, a, w); break;
    case EPI_CE_STATS: rc = dispatch<TM, EPI_CE_STATS>(c, ma, mb, mc, mp, a, w); break;
    case EPI_CE_DLOGITS: rc = dispatch<TM, EPI_CE_DLOGITS>(c, ma, mb, mc, mp, a, w); break;
    default: return fail("gemm: unknown epilogue");
  }
  if (rc != 0 || rest == 0) return rc;
  const dim3 grid(static_cast<unsigned>(rest * (2 * TM * BM / 8)));
  auto reduce = c.out_f32 ? pair_reduce_kernel<TM, true> : pair_reduce_kernel<TM, false>;
  CTB_CUDA_OK(launch_chained(a.chained != 0, reduce, grid, 256, 0, c.stream, 0, static_cast<const float*>(c.workspace), a, w, c.C,
                             c.ldc));
  return 0;
}

// -1: chosen by size; 0: never; 1: every plain product with enough tiles (CTB_GEMM_PAIR, ctb_gemm_set_pair).
inline int& pair_mode() {
  static int mode = [] {
    const char* e = std::getenv("CTB_GEMM_PAIR");
    return e != nullptr && (e[0] == '0' || e[0] == '1') ? e[0] - '0' : -1;
  }();
  return mode;
}

// Estimated times in microseconds, fitted to sustained runs of 277 products (the projections, their gradients and the
// head of five model widths, 80 to 16384 tokens) on B200s under their power cap; 5 % rms for the two-CTA forms, 7 % for the
// others.  A product is bound by the tensor core's chain of k-blocks in the busiest CTA, by the power that its
// multiplications draw (padding included), or by its operands' bytes, whichever is the longest: joined as a 5-norm.
double joined(double cycles, double flops, double rate, double bytes) {
  auto fifth = [](double x) { return x * x * x * x * x; };
  return std::pow(fifth(cycles / 1.8e3) + fifth(flops / rate / 1e9) + fifth(bytes / 5.5e6), 0.2);
}
long div_up(long a, long b) { return (a + b - 1) / b; }
double operand_bytes(const GemmCall& c) {
  return 2.0 * (static_cast<double>(c.M) * c.K + static_cast<double>(c.N) * c.K + static_cast<double>(c.M) * c.N);
}

double pair_time(const GemmCall& c, const PairPlan& p, int pairs) {
  const long num_k = div_up(c.K, 64), tiles = div_up(c.M, 256 * p.tm) * div_up(c.N, 256);
  const long rest = tiles - p.whole, units = p.whole + rest * p.slices;
  // the busiest pair: units go round robin, whole tiles first
  long k_blocks = 0, count = 0;
  for (const long pair : {0l, (units - 1) % pairs, p.whole > 0 ? (p.whole - 1l) % pairs : 0l, static_cast<long>(p.whole % pairs)}) {
    const long whole = p.whole > pair ? div_up(p.whole - pair, pairs) : 0;
    const long cut = (units > pair ? div_up(units - pair, pairs) : 0) - whole;
    const long mine = whole * num_k + cut * div_up(num_k, p.slices);
    if (mine > k_blocks || (mine == k_blocks && whole + cut > count)) {
      k_blocks = mine;
      count = whole + cut;
    }
  }
  const double idle = units < pairs ? 1.0 - static_cast<double>(units) / pairs : 0.0;
  const double cycles = k_blocks * (p.tm == 1 ? 482.0 : 930.0) * (1.0 + 0.1 * idle) + count * (p.tm == 1 ? 4600.0 : 8850.0);
  const double flops = 2.0 * tiles * 256 * p.tm * 256 * num_k * 64;
  const bool long_k = c.K > 5120;
  const double rate = p.tm == 1 ? (long_k ? 1.302 : 1.366) : (long_k ? 1.375 : 1.323);
  double t = 5.1 + joined(cycles, flops, rate, operand_bytes(c));
  if (rest > 0) t += 3.6 + rest * p.slices * p.tm * 524288.0 / 10.1e6;
  return t;
}

// The kernel that the product would go to otherwise (run_gemm, gemm_split_plan).
double one_cta_time(const GemmCall& c, int sms) {
  GemmCall sizes{};      // (of the sizes alone: the choice must not depend on which call came first)
  sizes.M = c.M; sizes.N = c.N; sizes.K = c.K; sizes.epi = c.epi; sizes.accumulate = c.accumulate;
  int width, slices;
  SplitCost cost;
  // 128-wide tiles: 0.28 us a k-block, not the 0.39 that the choice of the slices charges for both widths (240 products of 1
  // to 1400 tokens, 17 % rms; 35 x 256 x 32000 19 us, where 37 were expected and the two-CTA form took 29)
  if (gemm_split_plan(sizes, &width, &slices, &cost))
    return width == 128 ? 6.9 + 0.284 * cost.k_blocks : 0.76 + 1.131 * cost.cycles / 1.8e3;
  const long num_k = div_up(c.K, 64);
  const int tm = div_up(c.M, 256) * div_up(c.N, 256) >= 2l * sms ? 2 : 1;
  const long tiles = div_up(c.M, 128 * tm) * div_up(c.N, 256), rounds = div_up(tiles, sms);
  const double flops = 2.0 * tiles * 128 * tm * 256 * num_k * 64;
  const double rate = tm == 1 ? 1.26 : (c.K > 5120 ? 1.446 : 1.414);
  const double per_tile = num_k * (tm == 1 ? 688.0 : 1241.0) + (tm == 1 ? 2990.0 : 5990.0);
  return 5.4 + joined(rounds * per_tile, flops, rate, operand_bytes(c));
}

constexpr long MAX_WORKSPACE = 320l << 20;

}  // namespace gemm2

bool gemm_pair_forced() { return gemm2::pair_mode() == 1; }

long gemm_pair_workspace(const GemmCall& c, const PairPlan& p) {
  const long tiles = static_cast<long>((c.M + 256 * p.tm - 1) / (256 * p.tm)) * ((c.N + 255) / 256);
  return (tiles - p.whole) * p.slices * 256l * p.tm * 256l * 4l;
}

// Over the products of the fit the choice makes them 1.044 times as fast in the geometric mean, almost none more than 3 %
// slower than on the one-CTA kernels (the runs of one form differ by about 2 %).  Over 1614 others, of 1 to 16384 tokens, with
// operands out of memory and not run for long: 1.031 times, and 6 of the 1042 that take less than 40 us more than 3 % (and half a
// microsecond) slower.  It was 40 before the gain of a short product had to be 0.8 us, which is what the estimates of two
// short forms differ by without a reason (128 x 256 x 512: 7.9 us on one CTA and 8.6 on two, expected the other way round).
bool gemm_pair_plan(const GemmCall& c, PairPlan* plan) {
  using namespace gemm2;
  const int mode = pair_mode();
  if (mode == 0 || c.push.enabled || c.max_ctas > 0) return false;
  // a gathered operand: with flags only the persistent kernel will do, and without them (the pull was done
  // before the call) the product must come out the same
  if (c.gathered || c.a_flags != nullptr || c.b_flags != nullptr) return false;
  const int sms = sm_count(), pairs = sms / 2;
  const int num_n = (c.N + 255) / 256;
  // (whole bands of A stay in L2 while B goes by: 16 x 256 rows where they are no more than 42 MB)
  const int band = c.K <= 5120 ? 16 : 8;
  const PairPlan plain{1, (c.M + 255) / 256 * num_n, 1, band};
  if (mode == 1) {
    *plan = plain;
    return c.epi == EPI_STORE && c.bias == nullptr && plain.whole >= pairs && c.K >= 512;
  }
  // TMA stores whole 16 bytes: behind a row that ends inside of 16 it writes zeros, which the kernel for few tiles does not
  if (pairs < 1 || (c.epi == EPI_STORE && c.N % (c.out_f32 ? 4 : 8) != 0)) return false;
  struct Known {
    int m, n, k, form, found;
    PairPlan plan;
  };
  thread_local Known known[128] = {};      // the estimates take 2 us: a training step asks for the same few products
  const int form = 1 + (c.epi << 2) + (c.accumulate ? 2 : 0) + (c.out_f32 ? 1 : 0) + (sms << 8);
  Known& at = known[(static_cast<unsigned>(c.M) * 31u + static_cast<unsigned>(c.N) * 17u + static_cast<unsigned>(c.K) * 7u +
                     static_cast<unsigned>(form)) % 128u];
  if (at.form != form || at.m != c.M || at.n != c.N || at.k != c.K) {
    at = Known{c.M, c.N, c.K, form, 0, plain};
    const double other = one_cta_time(c, sms);
    double best = other < 16.0 ? other - 0.8 : 0.99 * other;
    auto consider = [&](const PairPlan& p) {
      const double t = pair_time(c, p, pairs);
      if (t >= best) return;
      best = t;
      at.plan = p;
      at.found = 1;
    };
    // whole tiles first: a wave that is nearly empty, or all of them where they are fewer than the pairs, may be split
    for (int tm = 1; tm <= 2; ++tm) {
      const int tiles = (c.M + 256 * tm - 1) / (256 * tm) * num_n;
      PairPlan p{tm, tiles, 1, band / tm};
      consider(p);
      if (c.epi != EPI_STORE || c.accumulate || tm * tiles > (1 << 20)) continue;
      for (int back = 0; back < 2; ++back) {
        p.whole = std::max(0, tiles / pairs - back) * pairs;
        for (p.slices = 2; p.slices <= 8 && (c.K + 63) / 64 >= 4 * p.slices; ++p.slices)
          if (p.whole < tiles && gemm_pair_workspace(c, p) <= MAX_WORKSPACE) consider(p);
      }
    }
  }
  *plan = at.plan;
  return at.found != 0;
}

int launch_gemm_pair(const GemmCall& c, const PairPlan& plan) {
  return plan.tm == 2 ? gemm2::run<2>(c, plan) : gemm2::run<1>(c, plan);
}

}  // namespace ctb

// 0: one-CTA kernels only; 1: plain products with enough tiles run on CTA pairs; -1: by size.  Returns the previous mode.
CTB_API int ctb_gemm_set_pair(int mode) {
  int& m = ctb::gemm2::pair_mode();
  const int before = m;
  m = mode < 0 ? -1 : (mode != 0 ? 1 : 0);
  return before;
}

// Which form of the two-CTA kernel a product takes by size: 1 and (row sub-tiles, whole tiles, slices, band), or 0.
CTB_API int ctb_gemm_pair_choice(int M, int N, int K, int out_f32, int accumulate, int* form) {
  ctb::GemmCall c{};
  c.M = M; c.N = N; c.K = K; c.out_f32 = out_f32; c.accumulate = accumulate; c.epi = ctb::EPI_STORE;
  ctb::PairPlan p;
  if (!ctb::gemm_pair_plan(c, &p)) return 0;
  form[0] = p.tm; form[1] = p.whole; form[2] = p.slices; form[3] = p.band;
  return 1;
}

// The same for the products of the loss: the statistics of the logits (kept or not), or with `gradients` their gradients.
CTB_API int ctb_ce_pair_choice(int rows, int vocab, int d, int gradients, int* form) {
  ctb::GemmCall c{};
  c.M = rows; c.N = vocab; c.K = d;
  c.epi = gradients ? ctb::EPI_CE_DLOGITS : ctb::EPI_CE_STATS;
  c.out_f32 = gradients ? 0 : 1;
  ctb::PairPlan p;
  if (!ctb::gemm_pair_plan(c, &p)) return 0;
  form[0] = p.tm; form[1] = p.whole; form[2] = p.slices; form[3] = p.band;
  return 1;
}

// The two-CTA kernel with a given plan, whatever the choice by size would be: for tests of every form that the plan may
// choose and for measurements of it.
CTB_API int ctb_gemm_pair(const void* A, const void* B, void* C, int M, int N, int K, long lda, long ldb, long ldc,
                          int a_mn, int b_mn, int out_f32, int accumulate, float alpha, const void* bias, int tm, int whole,
                          int slices, int band, void* workspace, long workspace_bytes, void* stream) {
  ctb::GemmCall c{};
  c.A = A; c.B = B; c.C = C; c.M = M; c.N = N; c.K = K; c.lda = lda; c.ldb = ldb; c.ldc = ldc;
  c.a_mn = a_mn; c.b_mn = b_mn; c.out_f32 = out_f32; c.accumulate = accumulate; c.alpha = alpha; c.bias = bias;
  c.epi = ctb::EPI_STORE; c.stream = stream; c.workspace = workspace;
  using ctb::fail;
  if (M <= 0 || N <= 0 || K <= 0) return fail("gemm_pair: M, N, K must be positive");
  if (lda % 8 || ldb % 8) return fail("gemm_pair: lda and ldb must be multiples of 8 elements (16 bytes)");
  if (ldc % (out_f32 ? 4 : 8) || reinterpret_cast<uintptr_t>(C) % 16) return fail("gemm_pair: rows of C must be 16-byte aligned");
  if ((tm != 1 && tm != 2) || band < 1) return fail("gemm_pair: tiles of 256 or 512 rows, bands of at least one");
  const ctb::PairPlan p{tm, whole, slices, band};
  const int tiles = ((M + 256 * tm - 1) / (256 * tm)) * ((N + 255) / 256);
  if (whole < 0 || whole > tiles || slices < 1 || (K + 63) / 64 < slices) return fail("gemm_pair: no such plan for this product");
  if (whole < tiles && accumulate) return fail("gemm_pair: split tiles are stored, not added");
  if (ctb::gemm_pair_workspace(c, p) > workspace_bytes) return fail("gemm_pair: workspace too small");
  return ctb::launch_gemm_pair(c, p);
}
