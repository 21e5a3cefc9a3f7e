// In-kernel NVLink collectives of the tensor-parallel path (sm_100a, peer-mapped symmetric memory).
//
// Activations between the projections are sharded by token rows over the tp ranks (rank t owns
// rows [t*Rl, (t+1)*Rl) of every [R, d] activation).  The collectives around the projections are
// therefore an all-gather of rows in front of a column-parallel GEMM and a reduce-scatter of rows
// behind a row-parallel GEMM:
//
//   tp_ag_pull     all-gather by pull.  Every rank keeps a *symmetric* [R, d] buffer and writes
//                  its own rows in place (the producing RMSNorm does); this kernel waits (bounded)
//                  for each peer's "rows ready" flag, copies that peer's rows out of the peer's
//                  buffer with 16-byte loads over NVLink and publishes one flag per chunk.  The
//                  tcgen05 GEMM acquires the chunk flags of exactly the A rows a tile reads
//                  (gemm.cu, a_flags) and starts on the rows this rank already owns, so transfer
//                  and math overlap tile by tile: together they are the fused all-gather -> GEMM.
//   (GEMM push)    the reduce-scatter half lives in the GEMM epilogue (gemm.cu, GemmPush): each
//                  partial-sum tile is stored straight into the owner's receive buffer.
//   tp_reduce      waits (bounded) for the push flags of all sources and sums the world slabs of
//                  this rank's rows in fp32, in rank order (deterministic).
//   ce_exchange    cross-rank half of the vocab-parallel cut cross-entropy: folds this rank's
//                  per-slab (max, sum-exp) and target logit, stores the three per-row numbers
//                  into every peer's statistics buffer, publishes a flag, waits (bounded) for the
//                  peers and combines them into the global log-sum-exp, the weighted NLL and the
//                  backward coefficient -- one launch, no host round trip.
//   embed_push     vocab-parallel embedding lookup: the rank that owns a token's embedding row
//                  stores it into the residual-stream buffer of the rank that owns the token.
//
// Peer memory is only ever touched with plain ld/st.  Every wait has a clock64() budget; on
// expiry the kernel records the site in the status word and returns.
//
// Reference counterpart: token_tiling.py:60,126,244 (all_gather / psum_scatter over tp),
// cut_cross_entropy.py:503-511 (pmax/psum over tp), runtime.py:334-338 (tp shardings).
#include <cuda_bf16.h>

#include "host_common.h"

namespace ctb {
namespace tpc {

constexpr int MAX_RANKS = 16;
constexpr int THREADS = 256;

struct Ptrs {
  void* p[MAX_RANKS];
};

enum : unsigned {
  SITE_TP_AG_READY = 0x0501,
  SITE_TP_REDUCE = 0x0502,
  SITE_TP_CE = 0x0503,
};

__device__ __forceinline__ uint4 ld_peer(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_sys(unsigned* p, unsigned v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait on one flag by thread 0 of the CTA; the verdict reaches every thread through the
// barrier itself.  No shared memory: a CTA of the pull kernel has to fit beside a resident
// tcgen05 GEMM CTA that owns nearly all of the SM's shared memory, or the GEMM would spin on
// flags that the pull can never get on the machine to publish.
__device__ __forceinline__ bool cta_wait_flag(const unsigned* f, unsigned epoch, long long budget, DeviceStatus* st,
                                              unsigned site, unsigned info) {
  int ok = 1;
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    while (ld_acquire_sys(f) < epoch) {
      if (clock64() - t0 > budget) {
        report_failure(st, site, info, epoch);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
  }
  return __syncthreads_and(ok) != 0;
}

// ------------------------------------------------------------------------------------------
// all-gather of token rows by pull, per-chunk flags for the consuming GEMM
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 4)
tp_ag_pull_kernel(Ptrs bufs, long slab_elems, int rank, int world, int chunk_elems, unsigned* __restrict__ flags,
                  unsigned epoch, const unsigned* __restrict__ ready, unsigned ready_epoch, long long budget,
                  DeviceStatus* st) {
  const int cps = static_cast<int>(slab_elems / chunk_elems);
  // own rows were written in place by the kernel before this one in stream order
  if (blockIdx.x == 0) {
    for (int c = threadIdx.x; c < cps; c += THREADS) st_release_gpu(flags + rank * cps + c, epoch);
  }
  const int total = cps * (world - 1);
  const int vec_per_chunk = chunk_elems / 8;
  __nv_bfloat16* mine = static_cast<__nv_bfloat16*>(bufs.p[rank]);
  int waited_src = -1;
  for (int pos = blockIdx.x; pos < total; pos += gridDim.x) {
    const int src = (rank + 1 + pos / cps) % world;
    const int c = pos % cps;
    if (src != waited_src) {
      if (!cta_wait_flag(ready + src, ready_epoch, budget, st, SITE_TP_AG_READY, static_cast<unsigned>(src)))
        return;
      waited_src = src;
    }
    const long off = static_cast<long>(src) * slab_elems + static_cast<long>(c) * chunk_elems;
    const uint4* from = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(bufs.p[src]) + off);
    uint4* to = reinterpret_cast<uint4*>(mine + off);
    for (int v = threadIdx.x; v < vec_per_chunk; v += THREADS * 8) {
      uint4 r[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = v + u * THREADS;
        if (i < vec_per_chunk) r[u] = ld_peer(from + i);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = v + u * THREADS;
        if (i < vec_per_chunk) to[i] = r[u];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      st_release_gpu(flags + src * cps + c, epoch);
    }
  }
}

// ------------------------------------------------------------------------------------------
// sum of the pushed partial slabs: out[r][c] = sum_src recv[src][r][c]   (+ optional residual)
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 4)
tp_reduce_kernel(const __nv_bfloat16* __restrict__ recv, long slab_elems, int world,
                 const unsigned* __restrict__ flags, unsigned epoch, __nv_bfloat16* __restrict__ out,
                 long long budget, DeviceStatus* st) {
  int bad = 0;
  if (threadIdx.x < world) {
    const long long t0 = clock64();
    while (ld_acquire_sys(flags + threadIdx.x) < epoch) {
      if (clock64() - t0 > budget) {
        report_failure(st, SITE_TP_REDUCE, static_cast<unsigned>(threadIdx.x), epoch);
        bad = 1;
        break;
      }
      __nanosleep(64);
    }
  }
  if (__syncthreads_or(bad)) return;
  const long nvec = slab_elems / 8;
  const long stride = static_cast<long>(gridDim.x) * THREADS;
  for (long v = blockIdx.x * static_cast<long>(THREADS) + threadIdx.x; v < nvec; v += stride) {
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = 0.f;
    for (int p = 0; p < world; ++p) {
      const uint4 raw = reinterpret_cast<const uint4*>(recv + static_cast<long>(p) * slab_elems)[v];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f2 = __bfloat1622float2(h[e]);
        s[2 * e] += f2.x;
        s[2 * e + 1] += f2.y;
      }
    }
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(s[2 * e], s[2 * e + 1]);
    reinterpret_cast<uint4*>(out)[v] = o;
  }
}

// ------------------------------------------------------------------------------------------
// vocab-parallel cut-CE: local slab fold -> exchange over peer memory -> global combine
// stats buffer of every rank: [world sources][3][rows_cap] fp32
// ------------------------------------------------------------------------------------------
struct CeExchangeArgs {
  const float* pmax;
  const float* psum;
  int slabs;
  const float* target_logit;      // zero where the target lies in another rank's vocabulary slice
  const float* weights;
  float grad_scale;
  float* lse;
  float* coef;
  float* block_nll;
  float* block_w;
  int rows;
  int rows_cap;
  int rank, world;
  Ptrs stats;                     // every rank's statistics buffer
  Ptrs flag;                      // &pads_of_rank_p[base + rank]
  const unsigned* my_flags;       // &my_pads[base]
  unsigned epoch;
  unsigned* counter;
  long long budget;
  DeviceStatus* status;
};

__device__ __forceinline__ float block_sum_256(float v, float* scratch) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x < 32) {
    t = threadIdx.x < THREADS / 32 ? scratch[threadIdx.x] : 0.f;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;  // valid in thread 0
}

__global__ void __launch_bounds__(THREADS, 2)
ce_exchange_kernel(const CeExchangeArgs a) {
  __shared__ float scratch[33];
  __shared__ int give_up;
  if (threadIdx.x == 0) give_up = 0;
  const long cap = a.rows_cap;
  // phase 1: fold this rank's slabs and store the row statistics into every rank's buffer
  for (int row = blockIdx.x * THREADS + threadIdx.x; row < a.rows; row += gridDim.x * THREADS) {
    float m = -INFINITY;
    for (int s = 0; s < a.slabs; ++s) m = fmaxf(m, a.pmax[static_cast<size_t>(s) * a.rows + row]);
    float acc = 0.f;
    for (int s = 0; s < a.slabs; ++s) {
      const size_t i = static_cast<size_t>(s) * a.rows + row;
      acc += a.psum[i] * __expf(a.pmax[i] - m);
    }
    const float tl = a.target_logit[row];
    for (int p = 0; p < a.world; ++p) {
      float* dst = static_cast<float*>(a.stats.p[p]) + static_cast<long>(a.rank) * 3 * cap;
      dst[row] = m;
      dst[cap + row] = acc;
      dst[2 * cap + row] = tl;
    }
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned done = atomicAdd(a.counter, 1u) + 1u;
    if (done == gridDim.x) {
      *a.counter = 0u;
      __threadfence_system();
      for (int p = 0; p < a.world; ++p) st_release_sys(static_cast<unsigned*>(a.flag.p[p]), a.epoch);
    }
  }
  // phase 2: wait for every source, combine
  if (threadIdx.x < a.world) {
    const long long t0 = clock64();
    while (ld_acquire_sys(a.my_flags + threadIdx.x) < a.epoch) {
      if (clock64() - t0 > a.budget) {
        report_failure(a.status, SITE_TP_CE, static_cast<unsigned>(threadIdx.x), a.epoch);
        give_up = 1;
        break;
      }
      __nanosleep(64);
    }
  }
  __syncthreads();
  float nll = 0.f, w = 0.f;
  if (!give_up) {
    const float* mine = static_cast<const float*>(a.stats.p[a.rank]);
    for (int row = blockIdx.x * THREADS + threadIdx.x; row < a.rows; row += gridDim.x * THREADS) {
      float m = -INFINITY;
      for (int p = 0; p < a.world; ++p) m = fmaxf(m, mine[static_cast<long>(p) * 3 * cap + row]);
      float acc = 0.f, tl = 0.f;
      for (int p = 0; p < a.world; ++p) {
        const float* src = mine + static_cast<long>(p) * 3 * cap;
        acc += src[cap + row] * __expf(src[row] - m);
        tl += src[2 * cap + row];
      }
      const float l = m + logf(acc);
      a.lse[row] = l;
      const float wt = a.weights[row];
      a.coef[row] = wt * a.grad_scale;
      w += wt;
      nll += (wt != 0.f) ? (l - tl) * wt : 0.f;
    }
  }
  const float bn = block_sum_256(nll, scratch);
  const float bw = block_sum_256(w, scratch);
  if (threadIdx.x == 0) {
    a.block_nll[blockIdx.x] = bn;
    a.block_w[blockIdx.x] = bw;
  }
}

// ------------------------------------------------------------------------------------------
// vocab-parallel embedding lookup: the owner of the embedding row stores it at the owner of the token
// ------------------------------------------------------------------------------------------
__global__ void embed_push_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table, Ptrs out,
                                  long tokens, int d, int vocab, int vocab_lo, int vocab_rows, int rows_per_rank) {
  const int nvec = d / 8;
  const long total = tokens * nvec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long t = i / nvec;
    const int v = static_cast<int>(i % nvec);
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    const int local = id - vocab_lo;
    if (local < 0 || local >= vocab_rows) continue;
    const int dest = static_cast<int>(t / rows_per_rank);
    const long row = t - static_cast<long>(dest) * rows_per_rank;
    reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(out.p[dest]) + row * d)[v] =
        reinterpret_cast<const uint4*>(table + static_cast<long>(local) * d)[v];
  }
}

// ------------------------------------------------------------------------------------------
// Embedding backward, deterministic: token gradients are summed per embedding row over runs of a
// stable sort of the ids (one CTA per run, fixed order, fp32) and added to the gradient table.
// Rows outside [vocab_lo, vocab_lo + vocab_rows) and the padding row are skipped.
// ------------------------------------------------------------------------------------------
// `sorted_ids` holds the token ids in order, `perm` where each came from; a run is a stretch of one id.  A CTA
// looks at EMB_WARPS positions and takes the runs that begin there, 32 * V columns a warp: short runs one
// per warp, runs longer than LONG_RUN (a mask token, a newline) by all eight warps together, whose partial sums
// are added in warp order, so the result does not depend on timing.  Finding the runs here instead of in a
// list spares the host a read back of their number.  With one CTA walking a run row by row, 4 bytes per
// load, 4000 repeats of one token were a chain of 4000 loads (968 us of a step).
// Bound by memory latency where runs are short: the ids and sources of the 8 positions and of the 23 behind them come in
// one load per lane, begins, lengths and sources of the runs are votes and shuffles, and the gradient row is requested
// with the first rows of the run.  With the positions tried one after the other, each a chain of loads, 8192 tokens of a
// 1536-wide table took 41 us for ids that occur once or twice and 32 for runs of 12; now 19 and 19.
constexpr int LONG_RUN = 16;
constexpr int EMB_WARPS = 8;
template <int V> struct EmbRaw;
template <> struct EmbRaw<8> { using T = uint4; };
template <> struct EmbRaw<2> { using T = uint32_t; };
template <typename G, int V>
__global__ void __launch_bounds__(EMB_WARPS * 32)
embedding_backward_kernel(const int* __restrict__ sorted_ids, const int* __restrict__ perm, int tokens,
                          const __nv_bfloat16* __restrict__ dout, G* __restrict__ grad, int d, int vocab_lo,
                          int vocab_rows, int pad_id) {
  using Raw = typename EmbRaw<V>::T;
  constexpr unsigned ALL = 0xffffffffu;
  __shared__ float part[EMB_WARPS][32 * V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.y * 32 + lane) * V;
  const bool live = c < d;
  const __nv_bfloat16* src = dout + (live ? c : 0);
  auto add = [&](const Raw& raw, float (&acc)[V]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < V / 2; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      acc[2 * e] += f.x;
      acc[2 * e + 1] += f.y;
    }
  };
  // this thread's columns of a gradient row, moved as whole 16-byte vectors where V = 8 (the launcher checks)
  constexpr int WORDS = V * static_cast<int>(sizeof(G)) / 4;
  auto row_at = [&](int local) { return grad + static_cast<long>(local) * d + c; };
  auto load_row = [&](const G* g, uint32_t (&w)[WORDS]) {
    if constexpr (WORDS % 4 == 0) {
#pragma unroll
      for (int i = 0; i < WORDS; i += 4) *reinterpret_cast<uint4*>(w + i) = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(g) + i);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) reinterpret_cast<G*>(w)[e] = g[e];
    }
  };
  auto add_row = [&](G* g, uint32_t (&w)[WORDS], const float (&acc)[V]) {
    G* v = reinterpret_cast<G*>(w);
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = static_cast<G>(static_cast<float>(v[e]) + acc[e]);
    if constexpr (WORDS % 4 == 0) {
#pragma unroll
      for (int i = 0; i < WORDS; i += 4) *reinterpret_cast<uint4*>(reinterpret_cast<uint32_t*>(g) + i) = *reinterpret_cast<const uint4*>(w + i);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) g[e] = v[e];
    }
  };
  // lane l: position first - 1 + l.  Lanes 1 to 8 are the positions of this CTA
  const int first = blockIdx.x * EMB_WARPS, p = first - 1 + lane;
  const bool in = p >= 0 && p < tokens;
  const int id = in ? __ldg(sorted_ids + p) : 0, from = in ? __ldg(perm + p) : 0;
  const int before = __shfl_up_sync(ALL, id, 1), beyond = __shfl_down_sync(ALL, id, LONG_RUN);
  const bool begins = in && lane >= 1 && lane <= EMB_WARPS && (p == 0 || before != id) && id != pad_id &&
                      id >= vocab_lo && id - vocab_lo < vocab_rows;
  const unsigned starts = __ballot_sync(ALL, begins);
  const unsigned longs = __ballot_sync(ALL, begins && p + LONG_RUN < tokens && beyond == id);
  if (((starts & ~longs) >> (warp + 1)) & 1u) {                  // (uniform in the warp)
    const int mine = __shfl_sync(ALL, id, warp + 1);
    const int n = __popc(__ballot_sync(ALL, in && id == mine));  // 1 to LONG_RUN, all of them in the window
    G* g = row_at(mine - vocab_lo);
    uint32_t old[WORDS];
    if (live) load_row(g, old);
    float acc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.f;
    constexpr int U = 8;
    for (int j = 0; j < n; j += U) {
      Raw raw[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int row = __shfl_sync(ALL, from, warp + 1 + j + k);
        if (j + k < n) raw[k] = __ldg(reinterpret_cast<const Raw*>(src + static_cast<long>(row) * d));
      }
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (j + k < n) add(raw[k], acc);
    }
    if (live) add_row(g, old, acc);
  }
  for (unsigned left = longs; left != 0u; left &= left - 1u) {   // (uniform in the CTA: every warp holds the same window)
    const int at = __ffs(left) - 1, mine = __shfl_sync(ALL, id, at), s0 = first - 1 + at;
    int s1 = s0 + LONG_RUN + 1, hi = tokens;                     // first position past the run, by bisection
    while (s1 < hi) {
      const int mid = s1 + (hi - s1) / 2;
      if (__ldg(sorted_ids + mid) == mine) s1 = mid + 1;
      else hi = mid;
    }
    float acc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.f;
    constexpr int U = 8;                                         // rows in flight; every eighth row of the run is this warp's
    for (int s = s0 + warp; s < s1; s += U * EMB_WARPS) {
      Raw raw[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        // past the end: the run's last row again, not added (unconditional loads stay in flight together)
        const int row = __ldg(perm + min(s + k * EMB_WARPS, s1 - 1));
        raw[k] = __ldg(reinterpret_cast<const Raw*>(src + static_cast<long>(row) * d));
      }
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (s + k * EMB_WARPS < s1) add(raw[k], acc);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) part[warp][e * 32 + lane] = acc[e];
    __syncthreads();
    if (warp == 0 && live) {
#pragma unroll 1
      for (int w = 1; w < EMB_WARPS; ++w)
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] += part[w][e * 32 + lane];
      G* g = row_at(mine - vocab_lo);
      uint32_t old[WORDS];
      load_row(g, old);
      add_row(g, old, acc);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------
// Token ids in ascending order, equal ones in the order of their positions (what a stable sort gives): one block sorts
// (id, position) pairs in shared memory, 64 bits each and no two alike, by a bitonic network.  For small micro-batches: a
// general stable sort and the conversions around it take 22.9 us of device time for 512 ids, 25.3 for 2048 and 28.4 for 4096,
// and some 40 us of host time, which is what bounds a step of that size; this takes 6.2, 18.0 and 36.3, one launch.
// A warp keeps to its own 64 slots for distances up to 32 and needs no block barrier there.
// ------------------------------------------------------------------------------------------
constexpr int SORT_MOST = 2048;
__global__ void __launch_bounds__(1024)
sort_ids_kernel(const int* ids, int words, int count, int slots, int* __restrict__ sorted_ids,
                int* __restrict__ perm) {
  let_successor_start();
  wait_for_predecessor();
  extern __shared__ unsigned long long sort_keys[];
  for (int i = threadIdx.x; i < slots; i += blockDim.x)
    sort_keys[i] = i < count ? (static_cast<unsigned long long>(static_cast<unsigned>(ids[static_cast<long>(i) * words]) ^ 0x80000000u) << 32) |
                                   static_cast<unsigned>(i)
                             : ~0ull;
  __syncthreads();
  for (int run = 2; run <= slots; run <<= 1) {
    for (int step = run >> 1; step > 0; step >>= 1) {
      const int t = threadIdx.x, lo = 2 * t - (t & (step - 1)), hi = lo + step;      // (a thread per pair)
      const unsigned long long a = sort_keys[lo], b = sort_keys[hi];
      if ((a > b) == ((lo & run) == 0)) {
        sort_keys[lo] = b;
        sort_keys[hi] = a;
      }
      if (step >= 64 || step == 1) __syncthreads();
      else __syncwarp();                               // this step and the next stay within the 64 slots of the warp's pairs
    }
  }
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    const unsigned long long key = sort_keys[i];
    sorted_ids[i] = static_cast<int>(static_cast<unsigned>(key >> 32) ^ 0x80000000u);
    perm[i] = static_cast<int>(static_cast<unsigned>(key));
  }
}

}  // namespace tpc
}  // namespace ctb

using namespace ctb;
using namespace ctb::tpc;

CTB_API int ctb_tp_ag_pull(void* const* buf_ptrs, long slab_elems, int rank, int world, int chunk_elems,
                           unsigned* flags, unsigned epoch, const unsigned* ready, unsigned ready_epoch, int ctas,
                           long long budget, void* stream) {
  if (world > MAX_RANKS) return fail("tp_ag_pull: too many ranks");
  if (chunk_elems % 8 || slab_elems % chunk_elems) return fail("tp_ag_pull: slab must be a whole number of chunks");
  Ptrs pp{};
  for (int i = 0; i < world; ++i) pp.p[i] = buf_ptrs[i];
  tp_ag_pull_kernel<<<ctas, THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      pp, slab_elems, rank, world, chunk_elems, flags, epoch, ready, ready_epoch, budget > 0 ? budget : CTB_SPIN_BUDGET,
      device_status());
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_tp_reduce(const void* recv, long slab_elems, int world, const unsigned* flags, unsigned epoch,
                          void* out, int ctas, long long budget, void* stream) {
  if (world > MAX_RANKS) return fail("tp_reduce: too many ranks");
  if (slab_elems % 8) return fail("tp_reduce: slab must be 16-byte aligned");
  tp_reduce_kernel<<<ctas, THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(recv), slab_elems, world, flags, epoch, static_cast<__nv_bfloat16*>(out),
      budget > 0 ? budget : CTB_SPIN_BUDGET, device_status());
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_ce_exchange_blocks(int rows) {
  const int want = (rows + THREADS - 1) / THREADS;
  const int cap = sm_count();
  return want < cap ? want : cap;
}

// block_nll / block_w must hold ctb_ce_exchange_blocks(rows) floats each.
CTB_API int ctb_ce_exchange(const float* pmax, const float* psum, int slabs, const float* target_logit,
                            const float* weights, float grad_scale, float* lse, float* coef, float* block_nll,
                            float* block_w, int rows, int rows_cap, int rank, int world, void* const* stats_ptrs,
                            unsigned* const* flag_ptrs, const unsigned* my_flags, unsigned epoch, unsigned* counter,
                            long long budget, void* stream) {
  if (world > MAX_RANKS) return fail("ce_exchange: too many ranks");
  if (rows > rows_cap) return fail("ce_exchange: more rows than the statistics buffers hold");
  CeExchangeArgs a{};
  a.pmax = pmax; a.psum = psum; a.slabs = slabs; a.target_logit = target_logit; a.weights = weights;
  a.grad_scale = grad_scale; a.lse = lse; a.coef = coef; a.block_nll = block_nll; a.block_w = block_w;
  a.rows = rows; a.rows_cap = rows_cap; a.rank = rank; a.world = world;
  for (int i = 0; i < world; ++i) {
    a.stats.p[i] = stats_ptrs[i];
    a.flag.p[i] = flag_ptrs[i];
  }
  a.my_flags = my_flags; a.epoch = epoch; a.counter = counter;
  a.budget = budget > 0 ? budget : CTB_SPIN_BUDGET; a.status = device_status();
  ce_exchange_kernel<<<ctb_ce_exchange_blocks(rows), THREADS, 0, static_cast<cudaStream_t>(stream)>>>(a);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_embed_push(const int* ids, const void* table, void* const* out_ptrs, int world, long tokens, int d,
                           int vocab, int vocab_lo, int vocab_rows, int rows_per_rank, void* stream) {
  if (world > MAX_RANKS) return fail("embed_push: too many ranks");
  if (d % 8) return fail("embed_push: hidden size must be a multiple of 8");
  Ptrs pp{};
  for (int i = 0; i < world; ++i) pp.p[i] = out_ptrs[i];
  const long work = tokens * (d / 8);
  long blocks = (work + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  embed_push_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      ids, static_cast<const __nv_bfloat16*>(table), pp, tokens, d, vocab, vocab_lo, vocab_rows, rows_per_rank);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// Token ids of a micro-batch in ascending order and where they came from, for the embedding gradient.  The ids may be 32- or
// 64-bit; of these the low word counts.  At most ctb_sort_ids_most() of them.
CTB_API int ctb_sort_ids_most() { return ctb::tpc::SORT_MOST; }
CTB_API int ctb_sort_ids(const void* ids, int id_bytes, long count, int* sorted_ids, int* perm, void* stream) {
  using namespace ctb::tpc;
  if (count <= 0) return 0;
  if (count > SORT_MOST || (id_bytes != 4 && id_bytes != 8)) return fail("sort_ids: at most 2048 ids of 32 or 64 bits");
  int slots = 64;
  while (slots < count) slots *= 2;
  CTB_CUDA_OK(launch_chained(true, sort_ids_kernel, 1, slots / 2, slots * sizeof(unsigned long long), stream, 0,
                             static_cast<const int*>(ids), id_bytes / 4, static_cast<int>(count), slots, sorted_ids, perm));
  return 0;
}

CTB_API int ctb_embedding_backward(const int* sorted_ids, const int* perm, long tokens, const void* dout, void* grad,
                                   int grad_f32, int d, int vocab_lo, int vocab_rows, int pad_id, void* stream) {
  if (tokens <= 0) return 0;
  if (d % 2) return fail("embedding_backward: hidden size must be even");
  if (tokens > 0x7fff0000L) return fail("embedding_backward: too many tokens");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto* src = static_cast<const __nv_bfloat16*>(dout);
  const int n = static_cast<int>(tokens);
  // whole 16-byte vectors of dout and of the table
  const bool wide = d % 8 == 0 && (reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(grad)) % 16 == 0;
  const int width = wide ? 256 : 64, chunks = (d + width - 1) / width;
  if (chunks > 65535) return fail("embedding_backward: hidden size too large");
  const dim3 grid(static_cast<unsigned>((n + EMB_WARPS - 1) / EMB_WARPS), static_cast<unsigned>(chunks));
#define CTB_EMB(G, V)                                                                                          \
  embedding_backward_kernel<G, V><<<grid, EMB_WARPS * 32, 0, s>>>(sorted_ids, perm, n, src, static_cast<G*>(grad), d, \
                                                                  vocab_lo, vocab_rows, pad_id)
  if (grad_f32) {
    if (wide) CTB_EMB(float, 8);
    else CTB_EMB(float, 2);
  } else {
    if (wide) CTB_EMB(__nv_bfloat16, 8);
    else CTB_EMB(__nv_bfloat16, 2);
  }
#undef CTB_EMB
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}
