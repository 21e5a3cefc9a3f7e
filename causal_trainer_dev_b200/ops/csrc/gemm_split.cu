// Plain products with too few output tiles to fill the GPU:  C[M,N] = A[M,K] * B[N,K]^T, the K range of
// every 128 x BN tile cut over the CTAs of one thread-block cluster.
//
// A down projection or an input gradient of a short batch (M = 1000, N = 1536, K = 17920) has 48
// tiles of 128 x 256: a third of the SMs work, each on a chain of K / 64 = 280 k-blocks, and nothing
// but K is left to divide.  Here a cluster of S = 2, 4 or 8 CTAs owns a tile; CTA s multiplies the
// k-blocks [s K/S, (s+1) K/S) into its own TMEM accumulator, writes the fp32 partial tile into its own
// shared memory (the operand ring is dead by then), and after one cluster barrier every CTA adds up 1/S
// of the rows over distributed shared memory and stores them.  No workspace, no atomics: the partial
// sums are added in the order of the slices, in fp32, so the result does not depend on timing.
//
//   warp 0       TMA producer (ring of 192 KiB, no multicast)
//   warp 1       single-thread tcgen05.mma issue;  warp 2 owns the TMEM allocation
//   warps 4-11   TMEM -> shared memory (two warpgroups, half of the columns each)
//   all warps    reduction and store
//
// Counterpart in the reference: XLA dot_general behind `linear`
// (src/causal_trainer/modeling/architecture.py:186-202).
#include "gemm.h"

#include <algorithm>

namespace ctb {
namespace gemm3 {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int THREADS = 384;
constexpr int MAX_SPLITS = 8;

enum : unsigned {
  SITE_S_PRODUCER_EMPTY = 0x0901,
  SITE_S_MMA_FULL = 0x0902,
  SITE_S_EPI_TFULL = 0x0903,
  SITE_S_DRAIN = 0x0904,
};

template <int BN>
struct Cfg {
  static constexpr int A_STAGE = BM * BK * 2;
  static constexpr int B_STAGE = BN * BK * 2;
  static constexpr int STAGES = 192 * 1024 / (A_STAGE + B_STAGE);
  static constexpr int OFF_B = STAGES * A_STAGE;
  static constexpr int OFF_BAR = OFF_B + STAGES * B_STAGE;
  static constexpr int BYTES = OFF_BAR + 256 + 1024;
  static_assert(BM * BN * 4 <= OFF_BAR, "the partial tile lies over the operand ring");
};

struct SplitArgs {
  int M, N, K;
  int splits;
  int out_f32;
  float alpha;
  const __nv_bfloat16* bias;
  void* C;
  long ldc;
  DeviceStatus* status;
  long long spin_budget;
  int chained;           // see launch_chained
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer(uint32_t addr, uint32_t rank) {
  uint32_t peer;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(peer)
               : "memory");
  return v;
}
// Byte offset of 16-byte chunk `chunk` of row `row` in a partial tile of `row_bytes` rows: the xor keeps
// both the row-per-thread writes and the chunk-per-thread reads off each other's banks.
__device__ __forceinline__ uint32_t partial_offset(uint32_t row, uint32_t chunk, uint32_t row_bytes) {
  return row * row_bytes + ((chunk ^ (row & 7u)) << 4);
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const SplitArgs args) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* empty = full + C::STAGES;
  uint64_t* tfull = empty + C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  const int S = args.splits;
  const int slice = static_cast<int>(cluster_rank());
  const int tile = blockIdx.x / S;
  const int num_m = (args.M + BM - 1) / BM;
  const int m0 = (tile % num_m) * BM, n0 = (tile / num_m) * BN;   // tiles that share B are neighbours
  const int num_k = (args.K + BK - 1) / BK;
  const int kb0 = num_k * slice / S, kb1 = num_k * (slice + 1) / S;   // never empty: S <= num_k
  DeviceStatus* st = args.status;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0u;
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (args.chained) let_successor_start();
  wait_for_predecessor();

  if (warp == 0) {
    {
      const uint32_t on = elect_one();         // the whole warp walks the k-blocks, one lane issues
      uint32_t stage = 0, phase = 0, armed = 0, armed_par = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag, st, SITE_S_PRODUCER_EMPTY, args.spin_budget)) {
          ok = false;
          break;
        }
        mbar_expect_tx_if(on, &full[stage], C::A_STAGE + C::B_STAGE);
        armed |= 1u << stage;
        armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
        uint8_t* sa = smem + stage * C::A_STAGE;
        uint8_t* sb = smem + C::OFF_B + stage * C::B_STAGE;
        const int k0 = kb * BK;
        if (A_MN) {
#pragma unroll
          for (int a = 0; a < BM / 64; ++a) tma_load_2d_if(on, sa + a * 8192, &map_a, &full[stage], m0 + a * 64, k0);
        } else {
          tma_load_2d_if(on, sa, &map_a, &full[stage], k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int a = 0; a < BN / 64; ++a) tma_load_2d_if(on, sb + a * 8192, &map_b, &full[stage], n0 + a * 64, k0);
        } else {
          tma_load_2d_if(on, sb, &map_b, &full[stage], k0, n0);
        }
        if (++stage == C::STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (on && (!ok || *abort_flag)) {
        // leave no copy in flight: wait (bounded) for the last phase armed on each stage
        for (int s = 0; s < C::STAGES; ++s) {
          if (!(armed & (1u << s))) continue;
          const long long t0 = clock64();
          while (!mbar_try_wait(&full[s], (armed_par >> s) & 1u)) {
            if (clock64() - t0 > 20000000ll) {
              report_failure(st, SITE_S_DRAIN, static_cast<unsigned>(s), (armed_par >> s) & 1u);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    {
      const uint32_t on = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&full[stage], phase, abort_flag, st, SITE_S_MMA_FULL, args.spin_budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * C::A_STAGE);
        const uint32_t sb = smem_u32(smem + C::OFF_B + stage * C::B_STAGE);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t da = A_MN ? desc_mnmajor(sa, k, 8192) : desc_kmajor(sa, k);
          const uint64_t db = B_MN ? desc_mnmajor(sb, k, 8192) : desc_kmajor(sb, k);
          umma_bf16_if(on, tmem_base, da, db, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
        }
        umma_commit_if(on, &empty[stage]);
        if (++stage == C::STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit_if(on, tfull);
    }
  } else if (warp >= 4) {
    // ------------------------------ TMEM -> partial tile ------------------------------
    const int half = (warp - 4) >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const bool got = mbar_wait(tfull, 0, abort_flag, st, SITE_S_EPI_TFULL, args.spin_budget);
    if (__all_sync(0xffffffffu, got)) {
      tc_fence_after();
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld32(taddr + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(smem + partial_offset(row, c * 8 + j, BN * 4)) =
              make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
  __syncwarp();
  cluster_barrier();                     // every slice's partial tile is in its CTA's shared memory

  // ------------------------------ sum of the slices, 1 / S of the rows per CTA ------------------------------
  constexpr int CHUNKS = BN / 4;
  const int rows = BM / S;
  const uint32_t base = smem_u32(smem);
  if (*abort_flag == 0u) {
    // two items per step: the loads of both are in flight together
    constexpr int U = 2;
#pragma unroll 1
    for (int first = threadIdx.x; first < rows * CHUNKS; first += U * THREADS) {
      float4 part[U][MAX_SPLITS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int item = min(first + u * THREADS, rows * CHUNKS - 1);
        const uint32_t at = base + partial_offset(slice * rows + item / CHUNKS, item % CHUNKS, BN * 4);
#pragma unroll
        for (int s = 0; s < MAX_SPLITS; ++s)
          if (s < S) part[u][s] = ld_peer(at, s);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int item = first + u * THREADS;
        const int m = m0 + slice * rows + item / CHUNKS, n = n0 + (item % CHUNKS) * 4;
        if (item >= rows * CHUNKS || m >= args.M || n >= args.N) continue;
        float v[4] = {part[u][0].x, part[u][0].y, part[u][0].z, part[u][0].w};
#pragma unroll
        for (int s = 1; s < MAX_SPLITS; ++s)
          if (s < S) {
            v[0] += part[u][s].x;
            v[1] += part[u][s].y;
            v[2] += part[u][s].z;
            v[3] += part[u][s].w;
          }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (args.bias != nullptr && n + e < args.N) v[e] += __bfloat162float(args.bias[n + e]);
          v[e] *= args.alpha;
        }
        const size_t to = static_cast<size_t>(m) * args.ldc + n;
        const bool whole = n + 4 <= args.N;
        if (args.out_f32) {
          float* out = static_cast<float*>(args.C) + to;
          if (whole) {
            *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 3; ++e)
              if (n + e < args.N) out[e] = v[e];
          }
        } else {
          __nv_bfloat16* out = static_cast<__nv_bfloat16*>(args.C) + to;
          if (whole) {
            *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
          } else {
#pragma unroll
            for (int e = 0; e < 3; ++e)
              if (n + e < args.N) out[e] = __float2bfloat16(v[e]);
          }
        }
      }
    }
  }
  __syncwarp();
  cluster_barrier();                     // nobody leaves while a peer still reads its partial tile
}

template <int BN, bool A_MN, bool B_MN>
int launch(const TensorMap& ma, const TensorMap& mb, const SplitArgs& a, int tiles, cudaStream_t s) {
  auto kern = gemm_split_kernel<BN, A_MN, B_MN>;
  static int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    CTB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::BYTES));
    configured_dev = dev;
  }
  CTB_CUDA_OK(launch_chained(a.chained != 0, kern, tiles * a.splits, THREADS, Cfg<BN>::BYTES, s, a.splits, ma.map, mb.map, a));
  return 0;
}

template <int BN>
int dispatch(const GemmCall& c, const TensorMap& ma, const TensorMap& mb, const SplitArgs& a, int tiles) {
  cudaStream_t s = static_cast<cudaStream_t>(c.stream);
  if (!c.a_mn && !c.b_mn) return launch<BN, false, false>(ma, mb, a, tiles, s);
  if (!c.a_mn && c.b_mn) return launch<BN, false, true>(ma, mb, a, tiles, s);
  if (c.a_mn && c.b_mn) return launch<BN, true, true>(ma, mb, a, tiles, s);
  return launch<BN, true, false>(ma, mb, a, tiles, s);
}

}  // namespace gemm3

// Chooses tile width and slices from estimated cycles and compares with the persistent kernel.  The figures
// are fits to a sweep of 100 shapes on B200: a k-block takes about 700 cycles at either tile width (operand
// latency, not the tensor core, once few CTAs run), a launch 6000 beside its k-blocks with the persistent
// kernel and 14000 here, where the slices are exchanged.  Clusters of 8, 4 and 2 leave some SMs of a 148-SM
// part unused: 14, 32 and 72 of them run at a time.  Examples (us, persistent -> here): 64 x 1536 x 8960
// 49 -> 15, 333 x 1536 x 32000 199 -> 60, 1000 x 1536 x 17920 107 -> 62; 2000 x 1536 x 17920 stays (112, 111).
bool gemm_split_plan(const GemmCall& c, int* width, int* splits, SplitCost* cost) {
  if (c.epi != EPI_STORE || c.accumulate || c.push.enabled || c.max_ctas > 0) return false;
  // a gathered operand: with flags only the persistent kernel will do, and without them (the pull was done
  // before the call) the product must come out the same
  if (c.gathered || c.a_flags != nullptr || c.b_flags != nullptr) return false;
  if (reinterpret_cast<uintptr_t>(c.C) % 16 != 0) return false;
  if (c.bias != nullptr && c.out_f32) return false;      // the fp32 store of the persistent kernel takes no bias
  const long num_m = (c.M + 127) / 128, num_k = (c.K + 63) / 64, sms = sm_count();
  const long tiles = num_m * ((c.N + 255) / 256);
  if (tiles > sms) return false;
  double best = 0.9 * (static_cast<double>(num_k) * 700.0 + 6000.0);      // the estimate has to promise a tenth
  bool found = false;
  for (int bn = 128; bn <= 256; bn += 128) {
    const long t = num_m * ((c.N + bn - 1) / bn);
    for (int s = 2; s <= gemm3::MAX_SPLITS; s *= 2) {
      if (num_k < 4 * s) break;      // a slice shorter than the ring is all ramp
      const long at_once = s == 2 ? sms * 72 / 148 : (s == 4 ? sms * 32 / 148 : sms * 14 / 148);
      if (at_once < 1) break;
      const long waves = (t + at_once - 1) / at_once;
      const long slice = (num_k + s - 1) / s;
      const double cycles = waves * (static_cast<double>(slice) * 700.0 + 14000.0);
      if (cycles < best) {
        best = cycles;
        *width = bn;
        *splits = s;
        if (cost != nullptr) *cost = SplitCost{cycles, waves * slice};
        found = true;
      }
    }
  }
  return found;
}

int launch_gemm_split(const GemmCall& c, int width, int splits) {
  const TensorMap ma = c.a_mn ? get_tensor_map_2d(c.A, Elt::BF16, c.M, c.K, c.lda, 64, 64, true)
                             : get_tensor_map_2d(c.A, Elt::BF16, c.K, c.M, c.lda, 64, 128, true);
  if (!ma) return 1;
  const TensorMap mb = c.b_mn ? get_tensor_map_2d(c.B, Elt::BF16, c.N, c.K, c.ldb, 64, 64, true)
                             : get_tensor_map_2d(c.B, Elt::BF16, c.K, c.N, c.ldb, 64, width, true);
  if (!mb) return 1;
  gemm3::SplitArgs a{};
  a.M = c.M; a.N = c.N; a.K = c.K;
  a.splits = splits;
  a.chained = chained_call(c);
  a.out_f32 = c.out_f32;
  a.alpha = c.alpha;
  a.bias = static_cast<const __nv_bfloat16*>(c.bias);
  a.C = c.C;
  a.ldc = c.ldc;
  a.status = device_status();
  a.spin_budget = c.spin_budget > 0 ? c.spin_budget : CTB_SPIN_BUDGET;
  const int tiles = ((c.M + 127) / 128) * ((c.N + width - 1) / width);
  return width == 256 ? gemm3::dispatch<256>(c, ma, mb, a, tiles) : gemm3::dispatch<128>(c, ma, mb, a, tiles);
}

}  // namespace ctb

// The cluster kernel at a given tile width (128 or 256) and number of slices (2, 4 or 8), whatever the plan would
// say: for tests of every form that the plan may choose and for measurements of the plan.
CTB_API int ctb_gemm_split(const void* A, const void* B, void* C, int M, int N, int K, long lda, long ldb, long ldc,
                           int a_mn, int b_mn, int out_f32, float alpha, const void* bias, int width, int slices,
                           void* stream) {
  using ctb::fail;
  if (M <= 0 || N <= 0 || K <= 0) return fail("gemm_split: M, N, K must be positive");
  if (lda % 8 || ldb % 8) return fail("gemm_split: lda and ldb must be multiples of 8 elements (16 bytes)");
  if (ldc % (out_f32 ? 4 : 8) || reinterpret_cast<uintptr_t>(C) % 16)
    return fail("gemm_split: rows of C must be 16-byte aligned");
  if (bias != nullptr && out_f32) return fail("gemm_split: a biased product is stored as bf16");
  if ((width != 128 && width != 256) || (slices != 2 && slices != 4 && slices != 8))
    return fail("gemm_split: width 128 or 256, 2, 4 or 8 slices");
  if ((K + 63) / 64 < slices) return fail("gemm_split: every slice needs a k-block");
  ctb::GemmCall c{};
  c.A = A; c.B = B; c.C = C; c.M = M; c.N = N; c.K = K; c.lda = lda; c.ldb = ldb; c.ldc = ldc;
  c.a_mn = a_mn; c.b_mn = b_mn; c.out_f32 = out_f32; c.alpha = alpha; c.bias = bias;
  c.epi = ctb::EPI_STORE; c.stream = stream;
  return ctb::launch_gemm_split(c, width, slices);
}
