// Flash attention backward for sm_100a, two kinds of work items from one template, no atomics:
//
//   MODE_DKV  KV-tile-owned: a CTA owns 128 keys of one KV head and walks the 64-row query blocks
//             of every query head of the GQA group that can see them, two blocks per iteration.
//                 S^T = K Q^T          dP^T = V dO^T            (tcgen05, TMEM)
//                 P^T = exp2(S^T c - lse),  dS^T = P^T (dP^T - delta)   (registers; the per-query
//                 statistics arrive negated and in log2 units, ready for packed fma / add)
//                 dV += P^T dO         dK += dS^T Q             (tcgen05, TMEM accumulators)
//             The reduction over the group's query heads happens in the TMEM accumulators.
//   MODE_DQ   Q-tile-owned: a CTA owns 128 query rows of one query head and walks the
//             64-key blocks it can see, two per iteration:  S = Q K^T, dP = dO V^T,
//             dS = P (dP - delta), dQ += dS K.
//
// Structure of both: resident operand pair X (K,V or Q,dO), streamed pair Y (Q,dO or K,V) of
// 128 rows through TMA rings (three slots of Y1 = Q or K, two of Y2 = dO or V), four compute warpgroups that share every iteration
// (32 of its 128 columns each).  An iteration is two independent 64-row blocks, so block ranges and
// work lists keep their 64-row granularity.  P^T / dS go back into TMEM as bf16 pairs over the scores
// they were computed from and are the TMEM A operands of the accumulate MMAs (they never cross
// shared memory); the Y tiles are reused in place as MN-major B operands.
//
// What bounds it.  A 128 x 128 iteration costs the tensor core 4 x 518 cycles (dQ: 3 x 518; measured, a
// 128 x 64 score tile takes 390 and not 259: it is bound by its operands' shared memory reads), the
// exponentials 1024 cycles (16 / clk / SM).  So two 64-row blocks share a 128-column tile, and the fixed
// costs (barrier round trips, masks, TMEM latency) are paid once per 32 columns of a thread.  S and dP have
// separate barriers, so that the exponentials overlap the dP product and dS overlaps dV and the next S
// (order of the tensor core: dV(i) S(i+1) dK(i) dP(i+1); with room in TMEM for a second S buffer:
// S(i+1) dV(i) dK(i) dP(i+1)), and each of P and dS is published in two halves of 16 columns per
// thread, so that the accumulate MMAs start on the first half.  Y1 has three slots because S(i+1) wants its
// operand early while dK(i) still reads the one before (with two joint slots the products waited 1200
// cycles per iteration for copies).  One document of 16384 tokens, 8 / 2 heads, D = 128, cycles per
// iteration of a CTA: dK/dV 4509 with joint slots, 3840 with three, 2615 with the warp-uniform issue
// of elect_one() (64-column tiles: 2 x 2700); dQ 3540, 3032, 2047.  Whole kernels 1.24 -> 0.79 ms and
// 0.88 -> 0.56 ms.  Now the compute warps are the longer side (P 1300, dS 420, masks 400 cycles).
//
// The results of an item are staged in ring slots (the producer leaves it one of Y1, and for dK / dV one of Y2) and not in
// the resident tiles' place, which the next item's tiles take as soon as the last dP is done.
//
// Reference counterparts: causal_trainer_attention_dq / _dkv
// (src/causal_trainer/kernels/efficient_attention.py:985-1173, 1270-1436); the psum that
// follows the reference's dK/dV kernel is not needed on one GPU because the group is reduced
// in TMEM.
#include <type_traits>

#include "attention.h"

namespace ctb {
namespace attn {

constexpr int BWD_THREADS = 640;   // 4 service warps + 4 compute warpgroups
constexpr int Y1_SLOTS = 3;        // Q (DKV) or K (DQ): needed first, released last
constexpr int Y2_SLOTS = 2;        // dO (DKV) or V (DQ)
constexpr int COMPUTE_WARPS = 16;

enum : unsigned {
  SITE_B_PROD = 0x0301,
  SITE_B_MMA_X = 0x0302,
  SITE_B_MMA_Y = 0x0303,
  SITE_B_MMA_T = 0x0304,
  SITE_B_CW_S = 0x0305,
  SITE_B_CW_ACC = 0x0307,
  SITE_B_BASE = 0x0308,
  SITE_B_ITEM = 0x0309,
};

template <int D>
struct BwdSmem {
  static constexpr int HALVES = D / 64;
  static constexpr int XT = HALVES * 16384;   // 128-row resident tile
  static constexpr int YT = HALVES * 16384;   // streamed tile: two 64-row blocks
  static constexpr int OFF_X = 0;             // X1, X2
  static constexpr int OFF_Y1 = 2 * XT;
  static constexpr int OFF_Y2 = OFF_Y1 + Y1_SLOTS * YT;
  // statistics of the streamed queries (DKV): 128 x -delta beside each Y1 slot, 128 x -lse*log2(e)
  // beside each Y2 slot (dS is read after dV has released Y2, so -delta cannot live there)
  static constexpr int OFF_DELTA = OFF_Y2 + Y2_SLOTS * YT;
  static constexpr int OFF_LSE = OFF_DELTA + Y1_SLOTS * 512;
  static constexpr int OFF_BAR = OFF_LSE + Y2_SLOTS * 512;
  static constexpr int OFF_ITEMS = OFF_BAR + 256;   // answer of the work request, two work items
  static constexpr int BYTES = OFF_BAR + 512;       // no slack: the tiles need a 1024-byte aligned base (checked)
  static_assert(BYTES <= 232448, "shared memory of one CTA");
  // TMEM columns: S buffers, dP, accumulators.  A second S buffer where it fits into 512 columns.
  static constexpr int S_BUFS_DKV = 2 * 128 + 128 + 2 * D <= 512 ? 2 : 1;
  static constexpr int S_BUFS_DQ = 2;
};

struct BwdMaps {
  CUtensorMap q, k, v, dout, out1, out2;     // out1: dV (DKV) or dQ (DQ), out2: dK (DKV)
};

// One work item, resolved once by the producer warp and handed to the other roles through shared memory.
struct alignas(16) BwdItem {
  int mode;          // MODE_DKV, MODE_DQ, or -1: no more work
  int b, head;       // batch and head of X (kv head for DKV, query head for DQ; 0 for the gathered rows of grouped DQ)
  int hkv, kbatch;   // kv head and batch of the K / V / dK / dV tensors
  int x0;            // first row of the resident tiles
  int y_lo64;        // first 64-row block of the streamed operand
  int y_n64;         // their number (per head)
  int y_base;        // grouped: first row (DKV) or key (DQ) of the streamed operand
  int n_entry;       // 64-row blocks to visit
  int list;          // block-sparse: offset of the item's entries in it_list;  dK/dV in parts: index of its partial tiles,
                     // -1: the whole tile
  int first;         // dK/dV in parts: first entry of this one
};
static_assert(sizeof(BwdItem) == 48, "three 16-byte reads");

// Of the `parts` work items that a launch has for a key tile, as many have work as leave each `least` entries (see dkv_least);
// one alone stores its results as if there were no others.
__device__ __forceinline__ int dkv_parts_used(const BwdArgs& args, int n_entry) {
  return max(1, min(args.parts, n_entry / args.least));
}

// The 64-row query blocks that see the key tile kb of row b: [first, first + count).  Only the queries this rank holds,
// [q_off, q_off + Sq), are walked.
__device__ __forceinline__ void dkv_queries(const BwdArgs& args, int b, int kb, int& first, int& count) {
  const int at = b * (args.S / 128) + kb;
  const int qlo = max(args.q_lo[at], args.q_off), qhi = min(args.q_hi[at], args.q_off + args.Sq);
  first = qlo / 64;
  count = qhi > qlo ? (qhi + 63) / 64 - first : 0;
}

// (PARTS here and below: the launch has several work items per key tile.  A kernel of its own, because what it adds to the loops and
// the epilogue costs a long call half a percent)
template <int MODE, bool PARTS>
__device__ __forceinline__ BwdItem bwd_item(const BwdArgs& args, const int cta) {
  constexpr bool DKV = (MODE == MODE_DKV);
  const int group = args.Hq / args.Hkv;
  const int nb128 = args.S / 128;
  BwdItem w;
  w.mode = MODE;
  w.y_base = 0;
  w.list = 0;
  w.first = 0;
  if (args.grp.desc != nullptr) {
    // grouped MoBA (see GroupArgs): gathered rows of one group against the keys of its block, no masks.
    // X = the item's resident tile: 128 keys of the block (dK/dV) or 128 gathered rows (dQ);
    // Y = 64-row blocks of the group's gathered rows (dK/dV) or of the block's keys (dQ).
    const int4 gd = __ldg(args.grp.desc + cta);
    w.hkv = gd.x >> 16;
    w.kbatch = gd.x & 0xffff;
    w.b = DKV ? w.kbatch : 0;
    w.head = DKV ? w.hkv : 0;
    w.x0 = DKV ? gd.y : cta * 128;
    w.y_lo64 = 0;
    w.y_n64 = gd.w <= 0 ? 0 : (DKV ? gd.w / 64 : args.grp.block / 64);
    w.y_base = DKV ? gd.z : gd.y;
    w.n_entry = w.y_n64;
    if (gd.w <= 0) w.mode = -2;                        // unused capacity: nothing is written
    return w;
  }
  // The first part of every key tile, then the second ones, ...: side by side, the parts that have no work in a call of short documents
  // came ahead of tiles and dQ items that do (2 rows of 2048 in documents of 200, 14 / 2 heads, 65.6 us, in this order 46.8).
  const int tiles = args.Hkv * args.B * nb128;
  int idx = DKV && PARTS ? cta % tiles : cta;
  if (DKV) {
    w.head = idx % args.Hkv;      // kv head
    idx /= args.Hkv;
    w.b = idx % args.B;
    const int kb = idx / args.B;  // ascending: key blocks near the start see the most queries
    w.x0 = kb * 128;
    dkv_queries(args, w.b, kb, w.y_lo64, w.y_n64);
    w.n_entry = w.y_n64 * group;
    w.hkv = w.head;
    if (PARTS) {
      // whole iterations (two entries) to every part that has work
      const int part = cta / tiles, used = dkv_parts_used(args, w.n_entry), all = w.n_entry;
      if (part >= used) w.mode = -2;
      w.first = all * part / used & ~1;
      w.n_entry = (part + 1 < used ? all * (part + 1) / used & ~1 : all) - w.first;
      w.list = used > 1 ? cta % tiles * args.parts + part : -1;
    }
  } else {
    w.head = idx % args.Hq;       // query head
    idx /= args.Hq;
    w.b = idx % args.B;
    const int qb = args.Sq / 128 - 1 - idx / args.B;  // descending: late query blocks see the most keys
    w.x0 = qb * 128;                                  // row of the local Q / dO / dQ
    const int klo = args.kv_lo[w.b * nb128 + args.q_off / 128 + qb];
    const int khi = args.kv_hi[w.b * nb128 + args.q_off / 128 + qb];
    w.y_lo64 = klo / 64;
    w.y_n64 = khi > klo ? (khi + 63) / 64 - w.y_lo64 : 0;
    w.n_entry = w.y_n64;
    w.hkv = w.head / group;
  }
  w.kbatch = w.b;
  // Block-sparse routing: the (64-row block, head) pairs come from a list instead of a range.
  if (args.sp.it_list != nullptr) sparse_list(args.sp, cta, w.list, w.n_entry);
  return w;
}

// entry -> (64-row block of the streamed operand, query head).  Iteration i holds entries 2i and
// 2i + 1 in the two halves of its tile; an odd last half repeats the last entry, fully masked.
template <int MODE, bool PARTS>
__device__ __forceinline__ void bwd_entry(const BwdArgs& args, const BwdItem& w, int e, int& block, int& head) {
  const bool sparse = args.sp.it_list != nullptr;
  const int entry = sparse ? __ldg(args.sp.it_list + w.list + e) : 0;
  if (PARTS) e += w.first;
  block = sparse ? (entry & 0xffffff) : w.y_lo64 + e % w.y_n64;
  if (args.grp.desc != nullptr) head = 0;
  else if (MODE == MODE_DQ) head = w.head;
  else head = w.hkv * (args.Hq / args.Hkv) + (sparse ? (entry >> 24) : e / w.y_n64);
}

// What every role needs to find its way, besides the work item.
struct BwdShared {
  uint8_t* smem;
  uint64_t *x_full, *x_empty, *y1_full, *y1_empty, *y2_full, *y2_empty, *s_full, *dp_full, *p_full, *ds_full, *acc_full, *acc_empty;
  volatile uint32_t* abort_flag;
  DeviceStatus* st;
  long long budget;
  uint32_t tmem_base;
};

// Positions that go on from one work item to the next.  The two rings and the barriers of the iterations keep their
// phases; `items` counts the items with work.
struct BwdWalk {
  uint32_t y1_slot = 0, y1_phase = 0;     // Y1 ring
  uint32_t y2 = 0;                        // uses of the Y2 ring: slot y2 & 1, phase (y2 >> 1) & 1
  uint32_t iterations = 0;                // dP and dS
  uint32_t s_phase = 0;                   // bit u: phase of S buffer u (MMA warp: of its P, which dQ items have not)
  uint32_t items = 0;

  __device__ __forceinline__ void next_y1() {
    if (++y1_slot == Y1_SLOTS) {
      y1_slot = 0;
      y1_phase ^= 1u;
    }
  }
  __device__ __forceinline__ uint32_t y2_slot() const { return y2 & 1u; }
  __device__ __forceinline__ uint32_t y2_phase() const { return (y2 >> 1) & 1u; }
};

template <int D, int MODE>
struct BwdTmem {
  static constexpr int S_BUFS = MODE == MODE_DKV ? BwdSmem<D>::S_BUFS_DKV : BwdSmem<D>::S_BUFS_DQ;
  static constexpr uint32_t DP = S_BUFS * 128;
  static constexpr uint32_t ACC1 = DP + 128;       // dV (DKV) or dQ (DQ)
  static constexpr uint32_t ACC2 = ACC1 + D;       // dK (DKV)
};

// Resident tiles of an item (one lane).
template <int D, int MODE>
__device__ __forceinline__ void bwd_load_x(uint32_t on, const BwdShared& sh, const BwdMaps& maps, const BwdItem& w) {
  using L = BwdSmem<D>;
  constexpr bool DKV = (MODE == MODE_DKV);
  mbar_expect_tx_if(on, sh.x_full, 2 * L::XT);
  const CUtensorMap* mx1 = DKV ? &maps.k : &maps.q;
  const CUtensorMap* mx2 = DKV ? &maps.v : &maps.dout;
  const int xh = DKV ? w.hkv : w.head;
  const int xb = DKV ? w.kbatch : w.b;
#pragma unroll
  for (int hf = 0; hf < L::HALVES; ++hf) {
    tma_load_4d_if(on, sh.smem + L::OFF_X + hf * 16384, mx1, sh.x_full, hf * 64, xh, w.x0, xb);
    tma_load_4d_if(on, sh.smem + L::OFF_X + L::XT + hf * 16384, mx2, sh.x_full, hf * 64, xh, w.x0, xb);
  }
}

// ------------------------------ producer ------------------------------
// The streamed tiles of an item, then the ring slots that its epilogue stages its results in: a slot whose full barrier
// completes without a copy belongs to the epilogue, which frees it when the results have left.
template <int D, int MODE, bool PARTS>
__device__ __forceinline__ bool bwd_produce(uint32_t on, const BwdShared& sh, const BwdMaps& maps, const BwdArgs& args,
                                            const BwdItem& w, BwdWalk& at) {
  using L = BwdSmem<D>;
  constexpr bool DKV = (MODE == MODE_DKV);
  const bool grouped = args.grp.desc != nullptr;
  const int n_iter = (w.n_entry + 1) / 2;
  const CUtensorMap* my1 = DKV ? &maps.q : &maps.k;
  const CUtensorMap* my2 = DKV ? &maps.dout : &maps.v;
  const int ybatch = DKV ? w.b * (grouped ? 0 : 1) : w.kbatch;
  for (int it = 0; it < n_iter; ++it) {
    int y0[2], yh[2];
    size_t stat[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {              // the two 64-row halves of the tile
      int block;
      bwd_entry<MODE, PARTS>(args, w, min(2 * it + q, w.n_entry - 1), block, yh[q]);
      if (!DKV) yh[q] = w.hkv;
      y0[q] = w.y_base + block * 64 - (DKV ? args.q_off : 0);   // streamed queries are stored locally
      stat[q] = grouped ? static_cast<size_t>(y0[q])
                        : (static_cast<size_t>(w.b) * args.Hq + yh[q]) * args.Sq + y0[q];
    }
    auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, float* stat_dst, const float* stat_src) {
      mbar_expect_tx_if(on, bar, L::YT + (DKV ? 512 : 0));
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        // the per-query statistics of the block travel with it (256 B each, 256 B aligned)
        if (DKV) tma_load_1d_if(on, stat_dst + q * 64, stat_src + stat[q], 256, bar);
#pragma unroll
        for (int hf = 0; hf < L::HALVES; ++hf)
          tma_load_4d_if(on, dst + hf * 16384 + q * 8192, map, bar, hf * 64, yh[q], y0[q], ybatch);
      }
    };
    if (!mbar_wait_warp(&sh.y1_empty[at.y1_slot], at.y1_phase ^ 1u, sh.abort_flag, sh.st, SITE_B_PROD, sh.budget)) return false;
    load(sh.smem + L::OFF_Y1 + at.y1_slot * L::YT, my1, &sh.y1_full[at.y1_slot],
         reinterpret_cast<float*>(sh.smem + L::OFF_DELTA + at.y1_slot * 512), args.neg_delta);
    at.next_y1();
    const uint32_t slot2 = at.y2_slot();
    if (!mbar_wait_warp(&sh.y2_empty[slot2], at.y2_phase() ^ 1u, sh.abort_flag, sh.st, SITE_B_PROD, sh.budget)) return false;
    load(sh.smem + L::OFF_Y2 + slot2 * L::YT, my2, &sh.y2_full[slot2],
         reinterpret_cast<float*>(sh.smem + L::OFF_LSE + slot2 * 512), args.neg_lse2);
    ++at.y2;
  }
  if (!mbar_wait_warp(&sh.y1_empty[at.y1_slot], at.y1_phase ^ 1u, sh.abort_flag, sh.st, SITE_B_PROD, sh.budget)) return false;
  if (on) mbar_arrive(&sh.y1_full[at.y1_slot]);
  at.next_y1();
  if (DKV) {
    if (!mbar_wait_warp(&sh.y2_empty[at.y2_slot()], at.y2_phase() ^ 1u, sh.abort_flag, sh.st, SITE_B_PROD, sh.budget)) return false;
    if (on) mbar_arrive(&sh.y2_full[at.y2_slot()]);
    ++at.y2;
  }
  return true;
}

// ------------------------------ MMA issuer ------------------------------
// `switched`: the item before was of the other mode, whose accumulators lie where this one keeps its dP.
template <int D, int MODE>
__device__ __forceinline__ bool bwd_issue(uint32_t on, const BwdShared& sh, const BwdItem& w, BwdWalk& at, bool switched) {
  using L = BwdSmem<D>;
  using T = BwdTmem<D, MODE>;
  constexpr bool DKV = (MODE == MODE_DKV);
  constexpr int S_BUFS = T::S_BUFS;
  const int n_iter = (w.n_entry + 1) / 2;
  bool ok = true;
  if (n_iter > 0) {
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
    constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, false, true);
    const uint32_t x1 = smem_u32(sh.smem + L::OFF_X);
    const uint32_t x2 = smem_u32(sh.smem + L::OFF_X + L::XT);
    const uint32_t y1_at = smem_u32(sh.smem + L::OFF_Y1);
    const uint32_t y2_at = smem_u32(sh.smem + L::OFF_Y2);
    // address arithmetic, not arrays: a runtime index into a local array would go through local memory
    auto tmem_s = [&](int u) -> uint32_t { return sh.tmem_base + static_cast<uint32_t>(u) * 128u; };
    const uint32_t tmem_dp = sh.tmem_base + T::DP;
    // S or dP of the tile in `y`: both operands K-major
    auto product = [&](uint32_t d, uint32_t x, uint32_t y) {
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        umma_bf16_if(on, d, desc_kmajor(x + (k / 4) * 16384, k % 4), desc_kmajor(y + (k / 4) * 16384, k % 4), idesc_s,
                     k != 0 ? 1u : 0u);
    };
    // accumulator += (P^T or dS) Y as its halves arrive.  The bf16 pairs of the 16 columns of group kk
    // sit in the first 8 columns of the group's own 16-column slice of the fp32 buffer
    auto accumulate = [&](uint64_t* full, uint32_t parity, uint32_t acc, uint32_t a, uint32_t y, int it) -> bool {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (!mbar_wait_warp(&full[half], parity, sh.abort_flag, sh.st, SITE_B_MMA_T, sh.budget)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = half; kk < 8; kk += 2)
          umma_bf16_ts_if(on, acc, a + 16 * kk, desc_mnmajor(y, kk, 16384), idesc_acc, (it | kk) != 0 ? 1u : 0u);
      }
      return true;
    };
    // the epilogue of the last item with work has read the accumulators
    const uint32_t acc_parity = (at.items & 1u) ^ 1u;
    if (switched) ok = mbar_wait_warp(sh.acc_empty, acc_parity, sh.abort_flag, sh.st, SITE_B_MMA_T, sh.budget);
    ok = ok && mbar_wait_warp(sh.x_full, at.items & 1u, sh.abort_flag, sh.st, SITE_B_MMA_X, sh.budget);
    uint32_t slot_a = at.y1_slot;            // Y1 slot of the next dK / dQ (at.y1_slot: of the next S)
    uint32_t y2_a = at.y2;                   // Y2 use of the next dV (at.y2: of the next dP)
    auto next_s = [&](int it) -> bool {
      if (!mbar_wait_warp(&sh.y1_full[at.y1_slot], at.y1_phase, sh.abort_flag, sh.st, SITE_B_MMA_Y, sh.budget)) return false;
      tc_fence_after();
      product(tmem_s(it % S_BUFS), x1, y1_at + at.y1_slot * L::YT);
      umma_commit_if(on, &sh.s_full[it % S_BUFS]);
      at.next_y1();
      return true;
    };
    auto next_dp = [&](bool last) -> bool {
      const uint32_t slot = at.y2_slot();
      if (!mbar_wait_warp(&sh.y2_full[slot], at.y2_phase(), sh.abort_flag, sh.st, SITE_B_MMA_Y, sh.budget)) return false;
      tc_fence_after();
      product(tmem_dp, x2, y2_at + slot * L::YT);
      umma_commit_if(on, sh.dp_full);
      if (!DKV) umma_commit_if(on, &sh.y2_empty[slot]);          // V is read by this product alone
      if (last) umma_commit_if(on, sh.x_empty);                  // the resident tiles may be replaced
      ++at.y2;
      return true;
    };
    ok = ok && next_s(0) && next_dp(n_iter == 1);
    for (int it = 0; ok && it < n_iter; ++it) {
      const bool more = it + 1 < n_iter;
      const int u = it % S_BUFS;
      // with one S buffer the next scores overwrite P, which dV reads: in issue order, so no wait
      if (S_BUFS == 2 && more && !next_s(it + 1)) return false;
      if (it == 0 && !switched &&
          !mbar_wait_warp(sh.acc_empty, acc_parity, sh.abort_flag, sh.st, SITE_B_MMA_T, sh.budget))
        return false;
      if (DKV) {
        if (!accumulate(sh.p_full + 2 * u, (at.s_phase >> u) & 1u, sh.tmem_base + T::ACC1, tmem_s(u),
                        y2_at + (y2_a & 1u) * L::YT, it))
          return false;
        umma_commit_if(on, &sh.y2_empty[y2_a & 1u]);
        ++y2_a;
        at.s_phase ^= 1u << u;
      }
      if (S_BUFS == 1 && more && !next_s(it + 1)) return false;
      if (!accumulate(sh.ds_full, at.iterations & 1u, sh.tmem_base + (DKV ? T::ACC2 : T::ACC1), tmem_dp,
                      y1_at + slot_a * L::YT, it))
        return false;
      ++at.iterations;
      umma_commit_if(on, &sh.y1_empty[slot_a]);
      if (++slot_a == Y1_SLOTS) slot_a = 0;
      if (more) ok = next_dp(it + 2 == n_iter);
      else umma_commit_if(on, sh.acc_full);
    }
    ++at.items;
  }
  at.next_y1();              // the slots that the epilogue stages in
  if (DKV) ++at.y2;
  return ok;
}

// ------------------------------ compute warpgroups ------------------------------
// Four compute warpgroups work on every iteration together: warpgroup wg takes columns
// [32 wg, 32 wg + 32) of the tile, i.e. 32 columns of entry 2 it + wg / 2.
template <int D, int MODE, bool PARTS>
__device__ __forceinline__ bool bwd_compute(const BwdShared& sh, const BwdMaps& maps, const BwdArgs& args, const BwdItem& w,
                                            BwdWalk& at) {
  using L = BwdSmem<D>;
  using T = BwdTmem<D, MODE>;
  constexpr bool DKV = (MODE == MODE_DKV);
  constexpr int S_BUFS = T::S_BUFS;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const bool grouped = args.grp.desc != nullptr, sparse = args.sp.it_list != nullptr;
  const int b = w.b, head = w.head, hkv = w.hkv, x0 = w.x0;
  const int group = args.Hq / args.Hkv, nb64 = args.S / 64;
  const int n_entry = w.n_entry, n_iter = (n_entry + 1) / 2;
  const int* it_list = sparse ? args.sp.it_list + w.list : nullptr;
  const int wg = (warp - 4) >> 2;
  const int quad = warp & 3;
  const int r = quad * 32 + lane;
  const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
  // position in the whole sequence of this thread's row: a key (DKV) or a local query (DQ)
  const int xi = x0 + r + (DKV ? 0 : args.q_off);
  const int xi_local = x0 + r;
  const int row_seg = grouped ? 1 : args.seg[b * args.S + xi];
  // interval of visible columns (whole-sequence positions): see the mask below
  int row_a, row_b;
  if (grouped) {
    row_a = -(1 << 30);       // everything is visible: padding rows hold zeros and contribute zero
    row_b = 1 << 30;
  } else if (DKV) {
    row_a = args.first_q[b * args.S + xi];
    row_b = args.run_end[b * args.S + xi];
  } else {
    row_a = args.run_start[b * args.S + xi];
    row_b = (args.lim != nullptr) ? args.lim[b * args.S + xi] : xi;
  }
  const int row_start = sparse ? args.sp.doc_start[b * args.S + xi] : 0;
  // DKV: the document-relative block of this key is the bit every query column is tested for
  const int row_blk = (sparse && DKV) ? (xi - row_start) / args.sp.block : 0;
  float neg_lse2 = 0.f, neg_delta = 0.f;      // DQ: per-row statistics (stored negated, lse in log2 units)
  if (!DKV) {
    const size_t row = grouped ? static_cast<size_t>(xi_local) : (static_cast<size_t>(b) * args.Hq + head) * args.Sq + xi_local;
    neg_lse2 = args.neg_lse2[row];
    neg_delta = args.neg_delta[row];
  }
  bool ok = true;
  const uint64_t scale2 = pack_f32x2(args.scale_log2, args.scale_log2);
  const int mine = wg >> 1;               // half of the tile this warpgroup works on
  // dense walk: (block, head) advance without a division per iteration (the first step moves by one
  // entry for the warpgroups of the second half, the others by two)
  int walk_block = 0, walk_head = 0;
  auto advance = [&](int n) {
    walk_block += n;
    while (walk_block >= w.y_n64) {
      walk_block -= w.y_n64;
      ++walk_head;
    }
  };
  if (!sparse && n_entry > 0) advance(PARTS ? w.first + mine : mine);
  for (int it = 0; it < n_iter; ++it) {
    const int entry_at = 2 * it + mine;
    const bool real = entry_at < n_entry;
    int yb, hq;
    if (sparse) {
      const int entry = __ldg(it_list + min(entry_at, n_entry - 1));
      yb = entry & 0xffffff;
      hq = DKV ? hkv * group + (entry >> 24) : head;
    } else {
      yb = w.y_lo64 + walk_block;
      hq = DKV ? hkv * group + walk_head : head;
      advance(2);
    }
    const int y0 = yb * 64;                   // (grouped: relative to the group, and nothing is masked)
    const int base = y0 + 32 * (wg & 1);      // first column of this thread
    // ---- visibility of this row against its 32 columns, as a bit mask.  The keys a query sees
    // and the queries that see a key are both contiguous intervals (runs are contiguous):
    //   DQ   row = query xi,  columns = keys     [start[xi], lim[xi]]
    //   DKV  row = key xi,    columns = queries  [first_q[xi], end[xi]]
    // Most tiles are wholly visible: two compares, the mask itself only where some row needs it.
    unsigned vis = 0xffffffffu;
    const bool inside = real && row_seg != 0 && row_a <= base && row_b >= base + 31;
    if (sparse || !__all_sync(0xffffffffu, inside)) {
      vis = (row_seg == 0 || !real) ? 0u : (bits_from(row_a - base) & bits_upto(row_b - base));
      if (sparse && vis != 0u) {
        if (DKV) {
          if ((row_blk >> 5) >= args.sp.words) {
            vis = 0u;
          } else {
            // when every query of the block selected this key's block the selection adds nothing
            const unsigned aw = __ldg(args.sp.allsel + ((static_cast<size_t>(b) * args.Hq + hq) * nb64 + yb) * args.sp.words +
                                      (row_blk >> 5));
            if (!((aw >> (row_blk & 31)) & 1u)) {
              // per-query selection bit of this key's block, for the 32 columns of this thread
              const unsigned* col_sel = args.sp.sel + ((static_cast<size_t>(b) * args.Hq + hq) * args.S + base) * args.sp.words +
                                        (row_blk >> 5);
              const int bit = row_blk & 31;
              unsigned selbits = 0u;
#pragma unroll 4
              for (int e = 0; e < 32; ++e)
                selbits |= ((__ldg(col_sel + static_cast<size_t>(e) * args.sp.words) >> bit) & 1u) << e;
              vis &= selbits;
            }
          }
        } else {
          const SparseRow sr = sparse_row(args.sp, b, head, args.Hq, args.S, xi, row_start, y0, 64);
          const unsigned above = bits_from(sr.bound - base);               // keys >= bound
          vis &= (sr.v0 ? ~above : 0u) | (sr.v1 ? above : 0u);
        }
      }
    }
    const bool warp_all = __all_sync(0xffffffffu, vis == 0xffffffffu);
    // DKV: per-query statistics of this thread's 32 columns, staged beside the tile by the producer
    const ulonglong2* lse_col = reinterpret_cast<const ulonglong2*>(sh.smem + L::OFF_LSE + at.y2_slot() * 512) + 8 * wg;
    const ulonglong2* delta_col = reinterpret_cast<const ulonglong2*>(sh.smem + L::OFF_DELTA + at.y1_slot * 512) + 8 * wg;
    const int u = it % S_BUFS;
    const uint32_t s_at = sh.tmem_base + static_cast<uint32_t>(u) * 128u + lane_off + 32 * wg;
    const uint32_t dp_at = sh.tmem_base + T::DP + lane_off + 32 * wg;
    if (DKV) {
      // (the statistics were written by bulk copies: these waits make them visible to the thread)
      if (!mbar_wait_warp(&sh.y1_full[at.y1_slot], at.y1_phase, sh.abort_flag, sh.st, SITE_B_CW_S, sh.budget) ||
          !mbar_wait_warp(&sh.y2_full[at.y2_slot()], at.y2_phase(), sh.abort_flag, sh.st, SITE_B_CW_S, sh.budget)) {
        ok = false;
        break;
      }
    }
    if (!mbar_wait_warp(&sh.s_full[u], (at.s_phase >> u) & 1u, sh.abort_flag, sh.st, SITE_B_CW_S, sh.budget)) {
      ok = false;
      break;
    }
    // (the accumulate MMAs that read P^T / dS of the previous iteration from these buffers were issued
    // before the products that refilled them, and the tensor core completes MMAs in issue order)
    tc_fence_after();
    // MASKED = false is the path of a warp whose rows all see all 32 columns: no selects.
    float p[32];
    auto probabilities = [&](auto masked_tag) {
      constexpr bool MASKED = decltype(masked_tag)::value;
      uint32_t sc[32];
      tmem_ld32(s_at, sc);
      tmem_ld_wait();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pw[8];
#pragma unroll
        for (int e4 = 0; e4 < 4; ++e4) {                 // groups of four columns
          uint64_t l2[2];                                // negated statistics, two columns per word
          if (DKV) {
            const ulonglong2 lv = lse_col[half * 4 + e4];
            l2[0] = lv.x;
            l2[1] = lv.y;
          } else {
            l2[0] = l2[1] = pack_f32x2(neg_lse2, neg_lse2);
          }
          // p = exp2(s * scale - lse): two columns per packed instruction
#pragma unroll
          for (int pr = 0; pr < 2; ++pr) {
            const int e = half * 16 + e4 * 4 + pr * 2;
            const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(sc[e]), __uint_as_float(sc[e + 1])), scale2, l2[pr]);
            float xa, xb;
            unpack_f32x2(x2, xa, xb);
            float pa = fast_exp2(xa), pb = fast_exp2(xb);
            if (MASKED) {
              if (!((vis >> e) & 1u)) pa = 0.f;
              if (!((vis >> (e + 1)) & 1u)) pb = 0.f;
            }
            p[e] = pa;
            p[e + 1] = pb;
            if (DKV) pw[e4 * 2 + pr] = pack_bf16(pa, pb);
          }
        }
        if (DKV) {
          tmem_st8(s_at + 16 * half, pw);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.p_full[2 * u + half]);
        }
      }
    };
    if (warp_all) probabilities(std::false_type{});
    else probabilities(std::true_type{});
    if (!mbar_wait_warp(sh.dp_full, at.iterations & 1u, sh.abort_flag, sh.st, SITE_B_CW_S, sh.budget)) {
      ok = false;
      break;
    }
    tc_fence_after();
    uint32_t rd[32];
    tmem_ld32(dp_at, rd);
    tmem_ld_wait();
    // dS = p * (dP - delta)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t dw[8];
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        uint64_t dl[2];
        if (DKV) {
          const ulonglong2 dv = delta_col[half * 4 + e4];
          dl[0] = dv.x;
          dl[1] = dv.y;
        } else {
          dl[0] = dl[1] = pack_f32x2(neg_delta, neg_delta);
        }
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {
          const int e = half * 16 + e4 * 4 + pr * 2;
          const uint64_t d2 = add_f32x2(pack_f32x2(__uint_as_float(rd[e]), __uint_as_float(rd[e + 1])), dl[pr]);
          const uint64_t ds2 = mul_f32x2(pack_f32x2(p[e], p[e + 1]), d2);
          float da, db;
          unpack_f32x2(ds2, da, db);
          dw[e4 * 2 + pr] = pack_bf16(da, db);
        }
      }
      tmem_st8(dp_at + 16 * half, dw);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.ds_full[half]);
    }
    at.next_y1();
    ++at.y2;
    ++at.iterations;
    at.s_phase ^= 1u << u;
  }
  // the epilogue pairs the warpgroups: pair u converts accumulator u, each warpgroup half of it
  const int u = wg & 1;
  const int half = wg >> 1;
  const bool writes = DKV || (u == 0);
  // ---- epilogue: accumulators -> bf16 -> staging -> TMA store ----
  if (ok && n_iter > 0) {
    ok = mbar_wait_warp(sh.acc_full, at.items & 1u, sh.abort_flag, sh.st, SITE_B_CW_ACC, sh.budget);
    tc_fence_after();
  }
  // pair 0 stages in the Y1 slot, pair 1 in the Y2 slot that the producer leaves to the epilogue
  const uint32_t slot = u == 0 ? at.y1_slot : at.y2_slot();
  if (ok && writes)
    ok = mbar_wait_warp(u == 0 ? &sh.y1_full[slot] : &sh.y2_full[slot], u == 0 ? at.y1_phase : at.y2_phase(), sh.abort_flag,
                        sh.st, SITE_B_CW_ACC, sh.budget);
  const bool any_bad = named_bar_or(2 + u, 256, !ok);
  if (!any_bad && DKV && PARTS && w.list >= 0) {
    // one of several work items of its key tile: fp32, as the accumulators hold them, 512 bytes of 32 keys at a time
    float4* to = reinterpret_cast<float4*>(args.partial) + (static_cast<size_t>(w.list) * 2 + u) * (D / 4) * 128 + r;
    const uint32_t acc = sh.tmem_base + (u == 1 ? T::ACC2 : T::ACC1);
#pragma unroll 1
    for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
      uint32_t rr[32];
      if (n_iter > 0) {
        tmem_ld32(acc + lane_off + c * 32, rr);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) rr[e] = 0u;
      }
#pragma unroll
      for (int jj = 0; jj < 8; ++jj)
        to[(c * 8 + jj) * 128] = make_float4(__uint_as_float(rr[jj * 4]), __uint_as_float(rr[jj * 4 + 1]),
                                             __uint_as_float(rr[jj * 4 + 2]), __uint_as_float(rr[jj * 4 + 3]));
    }
  } else if (!any_bad && writes) {
    // DKV: warpgroup 0 stores dV, warpgroup 1 stores dK (scaled); DQ: warpgroup 0 stores dQ (scaled).
    const uint32_t acc = sh.tmem_base + ((DKV && u == 1) ? T::ACC2 : T::ACC1);
    const float mul = (DKV && u == 0) ? 1.f : args.scale;
    uint8_t* stage_buf = sh.smem + (u == 0 ? L::OFF_Y1 : L::OFF_Y2) + slot * L::YT;      // [HALVES][128 rows][128 B]
    // the two warpgroups of the pair convert half of the head dimension each
#pragma unroll 1
    for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
      uint32_t rr[32];
      if (n_iter > 0) {
        tmem_ld32(acc + lane_off + c * 32, rr);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) rr[e] = 0u;
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        uint4 v;
        v.x = pack_bf16(__uint_as_float(rr[jj * 8 + 0]) * mul, __uint_as_float(rr[jj * 8 + 1]) * mul);
        v.y = pack_bf16(__uint_as_float(rr[jj * 8 + 2]) * mul, __uint_as_float(rr[jj * 8 + 3]) * mul);
        v.z = pack_bf16(__uint_as_float(rr[jj * 8 + 4]) * mul, __uint_as_float(rr[jj * 8 + 5]) * mul);
        v.w = pack_bf16(__uint_as_float(rr[jj * 8 + 6]) * mul, __uint_as_float(rr[jj * 8 + 7]) * mul);
        *reinterpret_cast<uint4*>(stage_buf + (c / 2) * 16384 + sw128_offset(r, (c % 2) * 4 + jj)) = v;
      }
    }
    tc_fence_before();
    fence_proxy_async_smem();
    named_bar_sync(4 + u, 256);
    if (r == 0 && half == 0) {
      const CUtensorMap* mo = (DKV && u == 1) ? &maps.out2 : &maps.out1;
      const int oh = DKV ? hkv : head;
      const int ob = DKV ? w.kbatch : b;
#pragma unroll
      for (int hf = 0; hf < L::HALVES; ++hf) {
        // grouped dK / dV: the history part joins what the own-block pass stored (one CTA per tile, so the sum
        // does not depend on timing)
        if (DKV && grouped) tma_reduce_add_4d(mo, stage_buf + hf * 16384, hf * 64, oh, x0, ob);
        else tma_store_4d(mo, stage_buf + hf * 16384, hf * 64, oh, x0, ob);
      }
      tma_commit_group();
    }
  }
  if (n_iter > 0) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(sh.acc_empty);      // the next item may accumulate
    ++at.items;
  }
  if (!any_bad && writes && r == 0 && half == 0) {
    tma_wait_group_read<0>();
    mbar_arrive(u == 0 ? &sh.y1_empty[slot] : &sh.y2_empty[slot]);
  }
  at.next_y1();
  if (DKV) ++at.y2;
  return !any_bad;
}

// dK and dV of key tiles that several work items share: the sums of their parts in the order of the parts (so the same bits
// whatever the timing), scaled and rounded once.  A block takes 16 channels of one gradient of one tile, a thread one key.
// Bound by the reads, out of L2.
template <int D>
__global__ void __launch_bounds__(128) attn_bwd_sum_kernel(const BwdArgs args, __nv_bfloat16* __restrict__ dk, long dk_rs,
                                                           __nv_bfloat16* __restrict__ dv, long dv_rs) {
  let_successor_start();
  wait_for_predecessor();
  constexpr int CHUNKS = D / 16;
  const int chunk = blockIdx.x % CHUNKS, u = blockIdx.x / CHUNKS % 2, item = blockIdx.x / (2 * CHUNKS), r = threadIdx.x;
  const int head = item % args.Hkv, b = item / args.Hkv % args.B, kb = item / args.Hkv / args.B;
  int first, count;
  dkv_queries(args, b, kb, first, count);
  const int used = dkv_parts_used(args, count * (args.Hq / args.Hkv));
  if (used == 1) return;                     // stored by its one work item
  const float* from = args.partial +
                      ((static_cast<size_t>(item) * args.parts * 2 + u) * (D / 4) * 128 + chunk * 4 * 128 + r) * 4;
  float4 sum[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) sum[j] = load_streamed(from + j * 512);
#pragma unroll 4
  for (int p = 1; p < used; ++p) {
    from += 2 * D * 128;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 v = load_streamed(from + j * 512);
      sum[j].x += v.x;
      sum[j].y += v.y;
      sum[j].z += v.z;
      sum[j].w += v.w;
    }
  }
  const float mul = u == 0 ? 1.f : args.scale;
  uint4* to = reinterpret_cast<uint4*>((u == 0 ? dv : dk) + (static_cast<long>(b) * args.S + kb * 128 + r) * (u == 0 ? dv_rs : dk_rs) +
                                       head * D + chunk * 16);
#pragma unroll
  for (int j = 0; j < 4; j += 2)
    to[j / 2] = make_uint4(pack_bf16(sum[j].x * mul, sum[j].y * mul), pack_bf16(sum[j].z * mul, sum[j].w * mul),
                           pack_bf16(sum[j + 1].x * mul, sum[j + 1].y * mul), pack_bf16(sum[j + 1].z * mul, sum[j + 1].w * mul));
}

// MODES: MODE_DKV, MODE_DQ, or MODE_BOTH: work items [0, dkv_items) of the first kind, then those of the second.
//
// A CTA stays on its SM and takes over work items of the grid that have not started (cluster launch control): the
// resident tiles, the first scores and the results of neighbouring items overlap, where a CTA of its own for each pays for
// its start, its first copies and its last stores one after the other (about 7000 cycles, a quarter of the dQ item of a
// packed row).  The next item is requested when the last copies of the current one are issued, not earlier: an item
// that waits behind a long one could have run elsewhere.
template <int D, int MODES, bool PARTS>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ BwdMaps dkv_maps, const __grid_constant__ BwdMaps dq_maps,
                const __grid_constant__ BwdArgs dkv, const __grid_constant__ BwdArgs dq, const int dkv_items) {
  using L = BwdSmem<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const BwdArgs& any = MODES == MODE_DQ ? dq : dkv;
  if ((smem_u32(smem) & 1023u) != 0u) {              // (uniform) the swizzled tiles would not be where TMA writes them
    if (threadIdx.x == 0) report_failure(any.status, SITE_B_BASE, smem_u32(smem), 0u);
    return;
  }
  BwdShared sh;
  sh.smem = smem;
  sh.x_full = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  sh.x_empty = sh.x_full + 1;
  sh.y1_full = sh.x_empty + 1;
  sh.y1_empty = sh.y1_full + Y1_SLOTS;
  sh.y2_full = sh.y1_empty + Y1_SLOTS;
  sh.y2_empty = sh.y2_full + Y2_SLOTS;
  sh.s_full = sh.y2_empty + Y2_SLOTS;       // [2] S of buffer u ready
  sh.dp_full = sh.s_full + 2;              // dP ready
  sh.p_full = sh.dp_full + 1;              // [2][2] S buffer u: half h (columns [16 h, 16 h + 16) of every 32) of P^T written
  sh.ds_full = sh.p_full + 4;              // [2] half h of dS written
  sh.acc_full = sh.ds_full + 2;
  sh.acc_empty = sh.acc_full + 1;
  uint64_t* item_full = sh.acc_empty + 1;  // [2] work item u resolved
  uint64_t* item_empty = item_full + 2;    // [2] and read by the MMA warp and the compute warps
  uint64_t* answer_full = item_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(answer_full + 1);
  sh.abort_flag = tmem_slot + 1;
  static_assert((1 + 1 + 2 * Y1_SLOTS + 2 * Y2_SLOTS + 2 + 1 + 4 + 2 + 2 + 2 + 2 + 1) * 8 + 8 <= 256, "barrier block");
  const uint32_t answer = smem_u32(smem + L::OFF_ITEMS);
  BwdItem* items = reinterpret_cast<BwdItem*>(smem + L::OFF_ITEMS + 16);
  sh.st = any.status;
  sh.budget = any.spin_budget;
  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;

  auto resolve = [&](int cta) -> BwdItem {
    if (MODES == MODE_DKV || (MODES == MODE_BOTH && cta < dkv_items)) return bwd_item<MODE_DKV, PARTS>(dkv, cta);
    return bwd_item<MODE_DQ, false>(dq, MODES == MODE_BOTH ? cta - dkv_items : cta);
  };
  BwdItem w;
  if (threadIdx.x < 32) {
    if (lane == 0) {
      mbar_init(sh.x_full, 1);
      mbar_init(sh.x_empty, 1);
      for (int s = 0; s < Y1_SLOTS; ++s) {
        mbar_init(&sh.y1_full[s], 1);
        mbar_init(&sh.y1_empty[s], 1);
      }
      for (int s = 0; s < Y2_SLOTS; ++s) {
        mbar_init(&sh.y2_full[s], 1);
        mbar_init(&sh.y2_empty[s], 1);
      }
      mbar_init(sh.dp_full, 1);
      for (int u = 0; u < 2; ++u) {
        mbar_init(&sh.s_full[u], 1);
        mbar_init(&sh.p_full[2 * u], COMPUTE_WARPS);
        mbar_init(&sh.p_full[2 * u + 1], COMPUTE_WARPS);
        mbar_init(&sh.ds_full[u], COMPUTE_WARPS);
        mbar_init(&item_full[u], 1);
        mbar_init(&item_empty[u], 1 + COMPUTE_WARPS);
      }
      mbar_init(sh.acc_full, 1);
      mbar_init(sh.acc_empty, COMPUTE_WARPS);
      mbar_init(answer_full, 1);
      *sh.abort_flag = 0u;
      mbar_fence_init();
    }
    __syncwarp();
    wait_for_predecessor();
    w = resolve(static_cast<int>(blockIdx.x));
    // the resident tiles are on their way while TMEM is allocated (with Q in the forward kernel, a layer's forward
    // and backward: 8.00 -> 7.77 ms on one document of 32768 tokens, 1096 -> 1047 us on 8 image rows of 4096)
    if (w.mode >= 0 && w.n_entry > 0) {
      const uint32_t on = elect_one();
      if (w.mode == MODE_DKV) bwd_load_x<D, MODE_DKV>(on, sh, dkv_maps, w);
      else bwd_load_x<D, MODE_DQ>(on, sh, dq_maps, w);
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  sh.tmem_base = *tmem_slot;
  wait_for_predecessor();

  // the next work item, for the roles that are told of it
  uint32_t turn = 0;
  auto take = [&](BwdItem& item) -> bool {
    const uint32_t u = turn & 1u;
    const bool got = mbar_wait_warp(&item_full[u], (turn >> 1) & 1u, sh.abort_flag, sh.st, SITE_B_ITEM, sh.budget);
    if (!got) return false;
    const int4* from = reinterpret_cast<const int4*>(&items[u]);
    int4* to = reinterpret_cast<int4*>(&item);
#pragma unroll
    for (int i = 0; i < 3; ++i) to[i] = from[i];
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_empty[u]);
    ++turn;
    return item.mode >= 0;
  };

  if (warp == 0) {
    const uint32_t on = elect_one();            // the whole warp walks, one lane issues
    BwdWalk at;
    uint32_t requests = 0;
    bool ok = true, loaded = true;              // the first item's resident tiles are on their way
    while (ok) {
      if (w.mode != -2) {                       // (unused capacity of a grouped launch is not passed on)
        const uint32_t u = turn & 1u;
        ok = mbar_wait_warp(&item_empty[u], ((turn >> 1) & 1u) ^ 1u, sh.abort_flag, sh.st, SITE_B_ITEM, sh.budget);
        if (!ok) break;
        if (lane == 0) {
          items[u] = w;
          mbar_arrive(&item_full[u]);
        }
        ++turn;
        if (w.mode < 0) break;
        if (w.n_entry > 0) {
          if (!loaded) {
            ok = mbar_wait_warp(sh.x_empty, (at.items & 1u) ^ 1u, sh.abort_flag, sh.st, SITE_B_PROD, sh.budget);
            if (!ok) break;
            if (w.mode == MODE_DKV) bwd_load_x<D, MODE_DKV>(on, sh, dkv_maps, w);
            else bwd_load_x<D, MODE_DQ>(on, sh, dq_maps, w);
          }
          ++at.items;
        }
        if (MODES != MODE_DQ && w.mode == MODE_DKV) ok = bwd_produce<D, MODE_DKV, PARTS>(on, sh, dkv_maps, dkv, w, at);
        else if (MODES != MODE_DKV) ok = bwd_produce<D, MODE_DQ, false>(on, sh, dq_maps, dq, w, at);
        if (!ok) break;
      }
      loaded = false;
      // a work item of the grid that has not started, if there is one
      mbar_expect_tx_if(on, answer_full, 16);
      work_request_if(on, answer, answer_full);
      ok = mbar_wait_warp(answer_full, requests & 1u, sh.abort_flag, sh.st, SITE_B_ITEM, sh.budget);
      if (!ok) break;
      ++requests;
      const int cta = work_answer(answer);
      fence_proxy_async_smem();                 // the next answer is written after this one is read
      __syncwarp();
      if (cta >= 0) w = resolve(cta);
      else w.mode = -1;
    }
    // not at the start: the successor's blocks would crowd on the SMs that run out of work first
    if (any.chained) let_successor_start();
  } else if (warp == 1) {
    const uint32_t on = elect_one();
    BwdWalk at;
    int mode = -1;
    while (take(w)) {
      const bool switched = mode >= 0 && mode != w.mode;
      bool ok = true;
      if (MODES != MODE_DQ && w.mode == MODE_DKV) ok = bwd_issue<D, MODE_DKV>(on, sh, w, at, switched);
      else if (MODES != MODE_DKV) ok = bwd_issue<D, MODE_DQ>(on, sh, w, at, switched);
      if (!ok) break;
      if (w.n_entry > 0) mode = w.mode;
    }
  } else if (warp >= 4) {
    BwdWalk at;
    while (true) {
      if (!take(w)) {
        // no more work; or this warp gave up on an item that another warp of the pair of warpgroups has, which waits for
        // this vote
        named_bar_or(2 + ((warp >> 2) - 1) % 2, 256, true);
        break;
      }
      bool ok = true;
      if (MODES != MODE_DQ && w.mode == MODE_DKV) ok = bwd_compute<D, MODE_DKV, PARTS>(sh, dkv_maps, dkv, w, at);
      else if (MODES != MODE_DKV) ok = bwd_compute<D, MODE_DQ, false>(sh, dq_maps, dq, w, at);
      if (!ok) break;
    }
    tma_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (*sh.abort_flag) wait_out_copies();      // (nobody sets it any more)
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(sh.tmem_base, 512);
  }
}

// Maps, arguments and number of work items of one mode.
template <int D, int MODE>
int prepare_bwd(const BwdCall& c, BwdMaps* maps, BwdArgs* args, int* items) {
  const bool grouped = c.grp.desc != nullptr;
  const int Sq = grouped ? c.gathered_rows : (c.Sq > 0 ? c.Sq : c.S);
  auto make = [&](const void* base, int heads, long row_stride, int rows, int seq, int batches) -> TensorMap {
    const uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(heads), static_cast<uint64_t>(seq),
                              static_cast<uint64_t>(batches)};
    const uint64_t strides[3] = {static_cast<uint64_t>(D), static_cast<uint64_t>(row_stride),
                                 static_cast<uint64_t>(row_stride) * seq};
    const uint32_t box[4] = {64, 1, static_cast<uint32_t>(rows), 1};
    return get_tensor_map_4d(base, Elt::BF16, dims, strides, box, true);
  };
  constexpr bool DKV = (MODE == MODE_DKV);
  // Resident operands use 128-row boxes, streamed operands 64-row boxes.
  // grouped: Q / dO / dQ are the gathered rows (one batch, one head)
  const int qh = grouped ? 1 : c.Hq, qb = grouped ? 1 : c.B;
  const TensorMap mq = make(c.q, qh, c.q_row_stride, DKV ? 64 : 128, Sq, qb);
  const TensorMap mk = make(c.k, c.Hkv, c.k_row_stride, DKV ? 128 : 64, c.S, c.B);
  const TensorMap mv = make(c.v, c.Hkv, c.v_row_stride, DKV ? 128 : 64, c.S, c.B);
  const TensorMap mdo = make(c.dout, qh, c.do_row_stride, DKV ? 64 : 128, Sq, qb);
  const TensorMap mo1 = DKV ? make(c.dv, c.Hkv, c.dv_row_stride, 128, c.S, c.B)
                            : make(c.dq, qh, c.dq_row_stride, 128, Sq, qb);
  const TensorMap mo2 = DKV ? make(c.dk, c.Hkv, c.dk_row_stride, 128, c.S, c.B) : mo1;
  if (!mq || !mk || !mv || !mdo || !mo1 || !mo2) return 1;
  BwdArgs a{};
  a.B = c.B; a.S = c.S; a.Hq = c.Hq; a.Hkv = c.Hkv;
  a.Sq = Sq; a.q_off = c.q_off;
  a.scale = c.scale;
  a.scale_log2 = c.scale * 1.4426950408889634f;
  a.seg = c.seg; a.lim = c.lim; a.kv_lo = c.kv_lo; a.kv_hi = c.kv_hi; a.q_lo = c.q_lo; a.q_hi = c.q_hi;
  a.run_start = c.run_start; a.run_end = c.run_end; a.first_q = c.first_q;
  a.neg_lse2 = c.neg_lse2; a.neg_delta = c.neg_delta;
  a.sp = c.sp;
  a.grp = c.grp;
  a.chained = !grouped && c.sp.it_list == nullptr && chained_rows(static_cast<long>(c.B) * Sq, c.Hq, D);
  a.status = device_status();
  a.spin_budget = c.spin_budget > 0 ? c.spin_budget : CTB_SPIN_BUDGET;
  a.parts = DKV && c.partial != nullptr ? c.parts : 1;
  a.least = c.least;
  a.partial = c.partial;
  *maps = BwdMaps{mq.map, mk.map, mv.map, mdo.map, mo1.map, mo2.map};
  *args = a;
  *items = grouped ? c.ctas : (DKV ? c.B * c.Hkv * (c.S / 128) * a.parts : c.B * c.Hq * (Sq / 128));
  return 0;
}

template <int D, int MODES, bool PARTS>
int launch_items_as(const BwdMaps& dkv_maps, const BwdMaps& dq_maps, const BwdArgs& dkv, const BwdArgs& dq, int dkv_items,
                 int dq_items, void* stream) {
  const int items = max(dkv_items, 0) + max(dq_items, 0);
  if (items == 0) return 0;
  auto kern = attn_bwd_kernel<D, MODES, PARTS>;
  static int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    CTB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdSmem<D>::BYTES));
    configured_dev = dev;
  }
  CTB_CUDA_OK(launch_chained((MODES == MODE_DQ ? dq : dkv).chained != 0, kern, items, BWD_THREADS, BwdSmem<D>::BYTES, stream, 0,
                             dkv_maps, dq_maps, dkv, dq, max(dkv_items, 0)));
  return 0;
}

template <int D, int MODES>
int launch_items(const BwdMaps& dkv_maps, const BwdMaps& dq_maps, const BwdArgs& dkv, const BwdArgs& dq, int dkv_items,
                 int dq_items, void* stream) {
  if (MODES != MODE_DQ && dkv.parts > 1)
    return launch_items_as<D, MODES == MODE_DQ ? MODE_DKV : MODES, true>(dkv_maps, dq_maps, dkv, dq, dkv_items, dq_items, stream);
  return launch_items_as<D, MODES, false>(dkv_maps, dq_maps, dkv, dq, dkv_items, dq_items, stream);
}

template <int D, int MODE>
int launch_bwd(const BwdCall& c) {
  BwdMaps maps;
  BwdArgs args{};
  int items = 0;
  if (prepare_bwd<D, MODE>(c, &maps, &args, &items)) return 1;
  return launch_items<D, MODE>(maps, maps, args, args, items, 0, c.stream);
}

// dK/dV as described by `dkv` and dQ as described by `dq`, in one launch: neither reads what the other writes, so the dQ
// work items fill the SMs that the last, long dK/dV items leave idle, and a short call pays for one launch less (8 image
// rows of 4096 tokens, 12 / 2 heads, forward and backward: 1014 -> 969 us; 2 rows of 256 tokens, with the launches' host
// side: 76 -> 38 us).
template <int D>
int launch_bwd_both(const BwdCall& dkv, const BwdCall& dq) {
  BwdMaps dkv_maps, dq_maps;
  BwdArgs dkv_args{}, dq_args{};
  int dkv_items = 0, dq_items = 0;
  if (prepare_bwd<D, MODE_DKV>(dkv, &dkv_maps, &dkv_args, &dkv_items)) return 1;
  if (prepare_bwd<D, MODE_DQ>(dq, &dq_maps, &dq_args, &dq_items)) return 1;
  return launch_items<D, MODE_BOTH>(dkv_maps, dq_maps, dkv_args, dq_args, dkv_items, dq_items, dkv.stream);
}

// Whether dQ shares memory with what the dK / dV items read of the queries (whole ranges: strided views that interleave
// count as sharing).
inline bool dq_over_inputs(const BwdCall& c) {
  const long rows = static_cast<long>(c.B) * c.Sq, width = static_cast<long>(c.Hq) * c.D;
  auto range = [&](const void* p, long row_stride, uintptr_t* from) {
    *from = reinterpret_cast<uintptr_t>(p);
    return *from + 2 * static_cast<uintptr_t>((rows - 1) * row_stride + width);
  };
  uintptr_t dq, q, dout;
  const uintptr_t dq_end = range(c.dq, c.dq_row_stride, &dq), q_end = range(c.q, c.q_row_stride, &q),
                  dout_end = range(c.dout, c.do_row_stride, &dout);
  return (dq < q_end && q < dq_end) || (dq < dout_end && dout < dq_end);
}

// dQ in the place of Q or dO: a dQ item replaces rows that no other dQ item reads, but dK / dV items do, so these come
// first, in a launch of their own.
template <int D>
int launch_bwd_dense(const BwdCall& c) {
  int rc;
  if (dq_over_inputs(c)) {
    rc = launch_bwd<D, MODE_DKV>(c);
    if (rc == 0) rc = launch_bwd<D, MODE_DQ>(c);
  } else {
    rc = launch_bwd_both<D>(c, c);
  }
  if (rc != 0 || c.partial == nullptr) return rc;
  BwdArgs a{};
  a.B = c.B; a.S = c.S; a.Hq = c.Hq; a.Hkv = c.Hkv;
  a.Sq = c.Sq; a.q_off = c.q_off;
  a.q_lo = c.q_lo; a.q_hi = c.q_hi;
  a.scale = c.scale;
  a.parts = c.parts;
  a.least = c.least;
  a.partial = c.partial;
  CTB_CUDA_OK(launch_chained(chained_rows(static_cast<long>(c.B) * c.Sq, c.Hq, D), attn_bwd_sum_kernel<D>,
                             c.B * c.Hkv * (c.S / 128) * 2 * (D / 16), 128, 0, c.stream, 0, a,
                             static_cast<__nv_bfloat16*>(c.dk), c.dk_row_stride, static_cast<__nv_bfloat16*>(c.dv),
                             c.dv_row_stride));
  return 0;
}

// Work items per key tile of dK/dV.  A key tile's item walks the queries of its whole group of heads, so a call with few
// key tiles (short rows, few kv heads) ends with a few SMs on the long ones of them: one row of 2048 tokens, 14 / 2 heads, has 32,
// and the longest is 112 iterations where an SM has 29 of the whole call.  The estimate (cycles) takes the rows for whole
// documents: an iteration of dK/dV 2615 and of dQ 2047, the start and end of an item 10000 and 8000, of a further part with its
// fp32 tiles 12000, the sum of the parts 8000.  Rows of short documents, whose tiles stay whole or nearly so (dkv_least), pay for
// that: the launch of the sums and the parts without work are 2 to 3 us.  Backward, us, uncut and so: 2 rows of 2048, 14 / 2 heads,
// one document 170.4, 95.3, documents of 350 54.4, 48.2, of 200 41.0, 43.5, of 128 28.9, 31.8; 4 rows of 512, 8 / 2 heads, 34.9, 25.8, of
// 200 26.7, 24.2, of 128 18.2, 20.2; 1 row of 1024, 28 / 4 heads, of 200 37.2, 29.5.  What did not mend it: the sums by the last part of
// a tile to finish (one SM reads them all: 5 to 8 us a cut tile), a compact list of the items made by every CTA with the sums at its
// end (the sums in the compute warps' loop spill registers: 6 to 12 us).
inline int dkv_parts(int B, int S, int Sq, int Hq, int Hkv) {
  const double tiles = static_cast<double>(B) * Hkv * (S / 128), rows = static_cast<double>(B) * Hq * (Sq / 128);
  const double longest = static_cast<double>(Hq / Hkv) * (Sq / 128), seen = (Sq / 128 + 1) / 2.;
  const double all = tiles * (longest / 2 * 2615 + 10000) + rows * (seen * 2047 + 8000), sms = sm_count();
  const double whole = max(longest * 2615 + 10000, all / sms);
  int best = 1;
  double least = 0.83 * whole;
  for (int p = 2; p <= 16 && longest >= 2 * p; ++p) {
    const double t = max(longest / p * 2615 + 10000, (all + tiles * (p - 1) * 12000) / sms) + 8000;
    if (t < least) {
      least = t;
      best = p;
    }
  }
  return best;
}

// Entries that a part of a key tile has at least: half of what the parts of the longest tile of one document have, and two iterations
// (two entries each).  Cut finer, rows of short documents with tiles enough for the GPU pay for the ends of their items (backward,
// us, without parts, with two iterations and with this: 2 rows of 2048, 14 / 2 heads, documents of 128 30.6, 48.1, 35.9; 1 row, 28 /
// 4 heads, of 200 41.0, 50.6, 44.1).  Parts twice as long lose where tiles are few (1 row of 2048, 14 / 2 heads, documents of 350 47.2,
// here 35.2, uncut 53.8).
inline int dkv_least(int Sq, int Hq, int Hkv, int parts) { return max(4, Hq / Hkv * (Sq / 128) / 2 / parts); }

}  // namespace attn
}  // namespace ctb

// Bytes that a backward pass of these sizes would like for partial sums of dK/dV (see dkv_parts), 0: none.
CTB_API long ctb_attn_bwd_workspace(int B, int S, int Sq, int Hq, int Hkv, int D) {
  if (B <= 0 || S <= 0 || Sq <= 0 || Hkv <= 0 || Hq % Hkv || (D != 64 && D != 128)) return 0;
  const int parts = ctb::attn::dkv_parts(B, S, Sq, Hq, Hkv);
  return parts > 1 ? static_cast<long>(B) * Hkv * (S / 128) * parts * 2 * 128 * D * 4 : 0;
}

// Whole backward of the queries [q_off, q_off + Sq) of every row (all of them: q_off 0, Sq = S): q / out / dout / dq, lse,
// neg_lse2 and neg_delta hold those queries; k / v / dk / dv cover all S keys (with fewer queries dk / dv are partial sums).
// The statistics are computed from out and lse first, unless out is null: then the caller hands them in.
// With less workspace than ctb_attn_bwd_workspace says, dK/dV of a key tile are one work item each, however few there are.
CTB_API int ctb_attn_bwd_range(const void* q, const void* k, const void* v, const void* out, const void* dout,
                               const float* lse, void* dq, void* dk, void* dv, float* neg_lse2, float* neg_delta,
                               const int* seg, const int* lim, const int* kv_lo, const int* kv_hi, const int* q_lo,
                               const int* q_hi, const int* run_start, const int* run_end, const int* first_q, int B, int S,
                               int Sq, int q_off, int Hq, int Hkv, int D, long q_rs, long k_rs, long v_rs, long o_rs,
                               long do_rs, long dq_rs, long dk_rs, long dv_rs, float scale, long long spin_budget,
                               void* workspace, long workspace_bytes, void* stream) {
  if (S % 128 || Sq % 128 || q_off % 128 || q_off < 0 || q_off + Sq > S)
    return ctb::fail("attention: S, Sq and q_off must be multiples of 128 with q_off + Sq <= S");
  if (Hq % Hkv) return ctb::fail("attention: Hq must be a multiple of Hkv");
  if (D != 64 && D != 128) return ctb::fail("attention: head_dim must be 64 or 128");
  if (out != nullptr) {
    const int rc = ctb_attn_bwd_stats(out, dout, lse, neg_lse2, neg_delta, B, Sq, Hq, D, o_rs, do_rs, stream);
    if (rc != 0) return rc;
  }
  ctb::attn::BwdCall c{};
  c.q = q; c.k = k; c.v = v; c.dout = dout; c.dq = dq; c.dk = dk; c.dv = dv; c.neg_lse2 = neg_lse2; c.neg_delta = neg_delta;
  c.seg = seg; c.lim = lim; c.kv_lo = kv_lo; c.kv_hi = kv_hi; c.q_lo = q_lo; c.q_hi = q_hi;
  c.run_start = run_start; c.run_end = run_end; c.first_q = first_q;
  c.B = B; c.S = S; c.Sq = Sq; c.q_off = q_off; c.Hq = Hq; c.Hkv = Hkv; c.D = D;
  c.q_row_stride = q_rs; c.k_row_stride = k_rs; c.v_row_stride = v_rs; c.do_row_stride = do_rs;
  c.dq_row_stride = dq_rs; c.dk_row_stride = dk_rs; c.dv_row_stride = dv_rs;
  c.scale = scale; c.spin_budget = spin_budget; c.stream = stream;
  const long wanted = ctb_attn_bwd_workspace(B, S, Sq, Hq, Hkv, D);
  if (wanted > 0 && workspace != nullptr && workspace_bytes >= wanted && reinterpret_cast<uintptr_t>(workspace) % 16 == 0 &&
      ((reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) % 16 == 0 && dk_rs % 8 == 0 && dv_rs % 8 == 0)) {
    c.parts = ctb::attn::dkv_parts(B, S, Sq, Hq, Hkv);
    c.least = ctb::attn::dkv_least(Sq, Hq, Hkv, c.parts);
    c.partial = static_cast<float*>(workspace);
  }
  return D == 128 ? ctb::attn::launch_bwd_dense<128>(c) : ctb::attn::launch_bwd_dense<64>(c);
}

// Block-sparse (MoBA) backward: `it_off` has one entry per CTA plus one, in grid order
// (mode 0: (key tile ascending, batch, kv head); mode 1: (query tile descending, batch, head));
// `it_list` holds 64-row block indices, with the head's index inside its GQA group in bits 24+
// for mode 0.
CTB_API int ctb_attn_bwd_sparse(int mode, const void* q, const void* k, const void* v, const void* dout, void* dq,
                                void* dk, void* dv, const float* neg_lse2, const float* neg_delta, const int* seg,
                                const int* lim, const int* kv_lo, const int* kv_hi, const int* q_lo, const int* q_hi,
                                const int* run_start, const int* run_end, const int* first_q, const int* it_off, const int* it_cnt, int it_stride,
                                const int* it_list, const unsigned* sel, const unsigned* allsel, const int* doc_start,
                                int block, int words, int B, int S, int Hq, int Hkv, int D,
                                long q_rs, long k_rs, long v_rs, long do_rs, long dq_rs, long dk_rs, long dv_rs,
                                float scale, long long spin_budget, void* stream) {
  if (S % 128) return ctb::fail("attention: sequence length must be a multiple of 128");
  if (Hq % Hkv) return ctb::fail("attention: Hq must be a multiple of Hkv");
  if (block < 128) return ctb::fail("sparse attention: the routing block must hold at least 128 tokens");
  ctb::attn::BwdCall c{};
  c.q = q; c.k = k; c.v = v; c.dout = dout; c.dq = dq; c.dk = dk; c.dv = dv; c.neg_lse2 = neg_lse2; c.neg_delta = neg_delta;
  c.seg = seg; c.lim = lim; c.kv_lo = kv_lo; c.kv_hi = kv_hi; c.q_lo = q_lo; c.q_hi = q_hi;
  c.run_start = run_start; c.run_end = run_end; c.first_q = first_q;
  c.B = B; c.S = S; c.Hq = Hq; c.Hkv = Hkv;
  c.q_row_stride = q_rs; c.k_row_stride = k_rs; c.v_row_stride = v_rs; c.do_row_stride = do_rs;
  c.dq_row_stride = dq_rs; c.dk_row_stride = dk_rs; c.dv_row_stride = dv_rs;
  c.scale = scale; c.spin_budget = spin_budget; c.stream = stream;
  c.sp.it_off = it_off; c.sp.it_cnt = it_cnt; c.sp.it_stride = it_stride; c.sp.it_list = it_list; c.sp.sel = sel;
  c.sp.doc_start = doc_start;
  c.sp.allsel = allsel; c.sp.block = block; c.sp.words = words;
  using namespace ctb::attn;
  if (D == 128) return mode == 0 ? launch_bwd<128, MODE_DKV>(c) : launch_bwd<128, MODE_DQ>(c);
  if (D == 64) return mode == 0 ? launch_bwd<64, MODE_DKV>(c) : launch_bwd<64, MODE_DQ>(c);
  return ctb::fail("attention: head_dim must be 64 or 128");
}

// Grouped MoBA backward (see GroupArgs).  dK/dV: one CTA per (group, 128-key tile), `dkv_ctas` descriptors; dk / dv are
// [B,S,Hkv,D] views that hold the own-block gradients, and the history part is added to them (tiles of groups without
// rows are left alone).  dQ: one CTA per 128 gathered rows, gathered_rows / 128 descriptors; dqg is [gathered_rows, D].
// qg / dog / the statistics are the gathered rows ([gathered_rows, D] contiguous, [gathered_rows] fp32, padding rows zero).
CTB_API int ctb_attn_bwd_grouped(const void* qg, const void* k, const void* v, const void* dog, void* dqg,
                                 void* dk, void* dv, const float* neg_lse2_g, const float* neg_delta_g,
                                 const void* dkv_desc, int dkv_ctas, const void* dq_desc, int gathered_rows, int block, int B,
                                 int S, int Hkv, int D, long k_rs, long v_rs, long dk_rs, long dv_rs, float scale,
                                 long long spin_budget, void* stream) {
  if (S % 128 || block % 128 || block < 128) return ctb::fail("grouped attention: S and the block must be multiples of 128");
  if (gathered_rows <= 0 || gathered_rows % 256) return ctb::fail("grouped attention: gathered rows must be a positive multiple of 256");
  ctb::attn::BwdCall c{};
  c.q = qg; c.k = k; c.v = v; c.dout = dog; c.dq = dqg; c.dk = dk; c.dv = dv;
  c.neg_lse2 = neg_lse2_g; c.neg_delta = neg_delta_g;
  c.B = B; c.S = S; c.Hq = Hkv; c.Hkv = Hkv;
  c.q_row_stride = D; c.do_row_stride = D; c.dq_row_stride = D;
  c.k_row_stride = k_rs; c.v_row_stride = v_rs; c.dk_row_stride = dk_rs; c.dv_row_stride = dv_rs;
  c.scale = scale; c.spin_budget = spin_budget; c.stream = stream;
  c.grp.block = block; c.gathered_rows = gathered_rows;
  ctb::attn::BwdCall dkv = c, dq = c;
  dkv.grp.desc = static_cast<const int4*>(dkv_desc);
  dkv.ctas = dkv_ctas;
  dq.grp.desc = static_cast<const int4*>(dq_desc);
  dq.ctas = gathered_rows / 128;
  using namespace ctb::attn;
  if (D == 128) return launch_bwd_both<128>(dkv, dq);
  if (D == 64) return launch_bwd_both<64>(dkv, dq);
  return ctb::fail("attention: head_dim must be 64 or 128");
}
