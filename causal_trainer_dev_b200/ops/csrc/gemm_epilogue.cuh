// Epilogues of the tcgen05 GEMM kernels (gemm.cu, gemm_pair.cu): one warpgroup drains the 128 accumulator rows
// of a TMEM slot or of a part of its columns.
#pragma once
#include "gemm.h"

namespace ctb {
namespace gemm {

constexpr int BM = 128;            // rows of one accumulator (one TMEM slot of a CTA)
constexpr int BN = 256;            // its columns
constexpr int EPI_BUF = 128 * 128;     // staging block: 128 rows x 128 B

// Copies a staged 128 x 128 B block (128-byte swizzle) to `out` (row stride `ld` elements) with
// 16-byte stores: thread -> (row etid/8 + 16*i, 16-byte column etid%8), so a warp writes four
// full 128 B rows per step.  Kept out of line so its address arithmetic does not raise the
// register count of the whole kernel.
static __device__ __noinline__ void push_block(const uint8_t* buf, __nv_bfloat16* out, long ld, int etid, int rows_left,
                                        int cols_left) {
  const int j = etid & 7;
  if (j * 8 >= cols_left) return;
  out += static_cast<long>(etid >> 3) * ld + j * 8;
#pragma unroll 4
  for (int i = 0; i < 8; ++i) {
    const int r = (etid >> 3) + i * 16;
    if (r < rows_left)
      *reinterpret_cast<uint4*>(out + static_cast<long>(i) * 16 * ld) =
          *reinterpret_cast<const uint4*>(buf + sw128_offset(r, j));
  }
}

// The registers of a TMEM load that this wait completes; named as operands so that nothing computed from them
// moves above it.
__device__ __forceinline__ void tmem_loaded(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Stages one 128-byte row per lane in the warp's block and sends the block's 32 rows to (x, y) of `map`.  `stage` is the
// warp's 4 KiB of the first of BUFS staging buffers.  Every block that is staged is stored: with two buffers the wait lets
// the newest store go on reading, which is the other buffer's only if each of the last `staged` blocks sent one.
//
// WIDE: the warpgroup's four blocks leave as one box of 128 rows, between barriers `bar` of its own.  For bf16 tiles of 128 rows:
// a short product is bound by its stores, and four times as many cost it a tenth (4608 x 3584 x 263 17.7 us, wide 16.3).  In
// fp32, or with 256 rows a tile, the barriers cost more (6144 x 4096 x 367 in fp32 33.0, wide 38.6).
template <int BUFS, bool WIDE = false>
__device__ __forceinline__ void store_rows(const uint32_t (&w)[32], uint8_t* stage, uint32_t& staged, int lane,
                                           const CUtensorMap* map, int x, int y, bool add, bool first = true, uint32_t bar = 0) {
  uint8_t* buf = stage + (BUFS == 2 ? (staged & 1u) * EPI_BUF : 0u);
  if (lane == 0 && first) tma_wait_group_read<BUFS - 1>();      // the block may still be read by the store that used it last
  if (WIDE) named_bar_sync(bar, 128);
  else __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(buf + sw128_offset(lane, j)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
  fence_proxy_async_smem();
  if (WIDE) named_bar_sync(bar, 128);
  else __syncwarp();
  if (lane == 0 && first) {
    if (add) tma_reduce_add_2d(map, buf, x, y);
    else tma_store_2d(map, buf, x, y);
    tma_commit_group();
  }
  ++staged;
}

// fp32 columns [0, columns) of the COLS at `taddr`, times alpha, to rows y and columns x of `map`.
template <int COLS, int BUFS>
__device__ __forceinline__ void drain_f32(uint32_t taddr, float alpha, int columns, uint8_t* stage, uint32_t& staged, int lane,
                                          const CUtensorMap* map, int x, int y, bool add) {
  const int blocks = min(COLS / 32, (columns + 31) / 32);
  uint32_t r[32];
  tmem_ld32(taddr, r);
#pragma unroll 1
  for (int c = 0; c < blocks; ++c) {
    uint32_t w[32];
    tmem_loaded(r);
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
    if (c + 1 < blocks) tmem_ld32(taddr + (c + 1) * 32, r);      // on its way while this block is staged
    store_rows<BUFS>(w, stage, staged, lane, map, x + c * 32, y, add);
  }
}

// Drains the COLS columns at `taddr` (which carries the warp's lane quadrant) to rows [m_sub, m_sub + 128) and columns
// [n0, n0 + COLS).  `row` is the thread's row of the slot, `etid` its index in the warpgroup, `bar_stage` a named
// barrier of the warpgroup, `epi` its BUFS staging blocks and `staged` the running count of blocks staged.
//
// Each warp stages and stores its own 32 rows, without a barrier of the warpgroup, and the next columns are loaded while these
// are staged: 650 cycles for 64 columns (the copy out of shared memory of the block before last), 1050 with 128-row
// blocks and two barriers for each.  WIDE: bf16 blocks of 128 rows (store_rows; `map_c` then has boxes of 128 rows).
template <int EPI, int COLS, int BUFS, bool WIDE = false>
__device__ __forceinline__ void drain_slot(const GemmArgs& args, const CUtensorMap* map_c, uint32_t taddr, int n0, int m_sub,
                                           int row, int etid, uint32_t bar_stage, uint8_t* epi, uint32_t& staged,
                                           bool add_into_c) {
  if (COLS < BN && n0 >= args.N) return;      // the second half of a tile may lie behind the matrix
  const int grow = m_sub + row;
  const int lane = etid & 31, quad = etid >> 5;
  uint8_t* stage = epi + quad * 4096;
  const int y = m_sub + quad * 32;
  // All rows of the warp may, too: it has nothing to store, and so must stage nothing (store_rows).
  // (In the push epilogue and with wide blocks, whose tiles have no 128 rows without one, the four warps meet at barriers.)
  const bool wide = WIDE && EPI != EPI_CE_STATS && !args.out_f32;
  if (EPI != EPI_PUSH && !wide && y >= args.M) return;
  if (EPI == EPI_CE_STATS) {
    // Online softmax statistics of this 256-column slab for one row per thread.
    const int target = (grow < args.M) ? args.ce_targets[static_cast<long>(grow) * args.ce_target_step] : -1;
    float vmax = -INFINITY, vsum = 0.f, tlogit = 0.f;
    bool has_target = false;
    const int blocks = min(COLS / 32, (args.N - n0 + 31) / 32);
    if (!args.ce_keep) {
      // (a loop of its own: with the copy and the early load of the next one the short statistics take a tenth longer, 1100 x
      // 32000 x 512 68 us, here 62)
#pragma unroll 1
      for (int c = 0; c < blocks; ++c) {
        const int col0 = n0 + c * 32;
        uint32_t r[32];
        tmem_ld32(taddr + c * 32, r);
        tmem_ld_wait();
        float cmax = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float v = (col0 + j < args.N) ? __uint_as_float(r[j]) : -INFINITY;
          r[j] = __float_as_uint(v);
          cmax = fmaxf(cmax, v);
          if (col0 + j == target) {
            tlogit = v;
            has_target = true;
          }
        }
        const float nmax = fmaxf(vmax, cmax);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) s += __expf(__uint_as_float(r[j]) - nmax);
        vsum = vsum * __expf(vmax - nmax) + s;
        vmax = nmax;
      }
    } else {
      uint32_t r[32];
      tmem_ld32(taddr, r);
#pragma unroll 1
      for (int c = 0; c < blocks; ++c) {
        const int col0 = n0 + c * 32;
        float v[32];
        float cmax = -INFINITY;
        tmem_loaded(r);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          v[j] = (col0 + j < args.N) ? __uint_as_float(r[j]) : -INFINITY;
          cmax = fmaxf(cmax, v[j]);
          if (col0 + j == target) {
            tlogit = v[j];
            has_target = true;
          }
        }
        uint32_t w[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) w[j] = __float_as_uint(v[j]);
        if (c + 1 < blocks) tmem_ld32(taddr + (c + 1) * 32, r);
        store_rows<BUFS>(w, stage, staged, lane, map_c, col0, y, false);      // (columns behind the matrix are cut off)
        const float nmax = fmaxf(vmax, cmax);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) s += __expf(v[j] - nmax);
        vsum = vsum * __expf(vmax - nmax) + s;
        vmax = nmax;
      }
    }
    if (grow < args.M) {
      const int slab = n0 / BN;
      args.ce_max[static_cast<size_t>(slab) * args.M + grow] = vmax;
      args.ce_sum[static_cast<size_t>(slab) * args.M + grow] = vsum;
      if (has_target) args.ce_target_logit[grow] = tlogit;
    }
  } else if (args.out_f32) {
    drain_f32<COLS, BUFS>(taddr, args.alpha, args.N - n0, stage, staged, lane, map_c, n0, y, add_into_c);
  } else {
    float lse = 0.f, coef = 0.f;
    int target = -1;
    if (EPI == EPI_CE_DLOGITS && grow < args.M) {
      lse = args.ce_lse[grow];
      coef = args.ce_coef[grow];
      target = args.ce_targets[static_cast<long>(grow) * args.ce_target_step];
    }
    const int blocks = min(COLS / 64, (args.N - n0 + 63) / 64);
    uint32_t r[2][32];
    tmem_ld32(taddr, r[0]);
    tmem_ld32(taddr + 32, r[1]);
#pragma unroll 1
    for (int c = 0; c < blocks; ++c) {
      const int col0 = n0 + c * 64;
      uint32_t w[32];
      tmem_loaded(r[0]);
      tmem_loaded(r[1]);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int cb = col0 + hh * 32;
        if (EPI == EPI_CE_DLOGITS) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float pv = __expf(__uint_as_float(r[hh][j]) - lse);
            if (cb + j == target) pv -= 1.f;
            r[hh][j] = __float_as_uint(pv * coef);
          }
        } else if (args.bias != nullptr) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float bv = (cb + j < args.N) ? __bfloat162float(args.bias[cb + j]) : 0.f;
            r[hh][j] = __float_as_uint(__uint_as_float(r[hh][j]) + bv);
          }
        }
        if (args.alpha != 1.f) {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[hh][j] = __float_as_uint(__uint_as_float(r[hh][j]) * args.alpha);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j)
          w[hh * 16 + j] = pack_bf16(__uint_as_float(r[hh][2 * j]), __uint_as_float(r[hh][2 * j + 1]));
      }
      if (c + 1 < blocks) {      // on their way while this block is staged
        tmem_ld32(taddr + (c + 1) * 64, r[0]);
        tmem_ld32(taddr + (c + 1) * 64 + 32, r[1]);
      }
      if (EPI != EPI_PUSH) {
        store_rows<BUFS, WIDE>(w, stage, staged, lane, map_c, col0, WIDE ? m_sub : y, add_into_c, !WIDE || quad == 0, bar_stage);
      } else {
        // reduce-scatter by push: the warpgroup's 128 threads copy the staged 128 x 128 B block into the
        // owner's receive buffer with 16-byte stores (peer memory: plain st.global only)
        uint8_t* buf = epi + (BUFS == 2 ? (staged & 1u) * EPI_BUF : 0u);
        named_bar_sync(bar_stage, 128);      // the copies that read this block last are out
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(buf + sw128_offset(row, j)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        named_bar_sync(bar_stage, 128);
        if (m_sub < args.M) {
          const int grow0 = args.push.row_offset + m_sub;
          const int dest = grow0 / args.push.rows_per_rank;
          const long drow0 = static_cast<long>(args.push.src_rank) * args.push.rows_per_rank +
                             (grow0 - dest * args.push.rows_per_rank);
          push_block(buf, args.push.dest[dest] + drow0 * args.push.ld + col0, args.push.ld, etid,
                     args.M - m_sub, args.N - col0);
        }
        ++staged;
      }
    }
    if (EPI == EPI_PUSH && m_sub < args.M) {
      // this 128-row piece is on its way: count it, and publish the flag with the last one
      __threadfence_system();
      named_bar_sync(bar_stage, 128);
      if (etid == 0) {
        const int dest = (args.push.row_offset + m_sub) / args.push.rows_per_rank;
        const unsigned done = atomicAdd(args.push.counters + dest, 1u) + 1u;
        if (done == static_cast<unsigned>(args.push.tiles_per_dest)) {
          args.push.counters[dest] = 0u;
          __threadfence_system();
          asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(args.push.flag[dest]), "r"(args.push.epoch)
                       : "memory");
        }
      }
    }
  }
}

}  // namespace gemm
}  // namespace ctb
