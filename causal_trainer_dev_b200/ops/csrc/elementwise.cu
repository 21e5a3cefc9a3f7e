// Memory-bound kernels of the decoder layer and the optimizer (sm_100a, HBM3e bound):
// RMSNorm forward/backward (optional fused residual add), RoPE (in place on the packed QKV
// projection, both pairings, partial rotary, arbitrary positions), SwiGLU forward/backward
// on the packed gate|up projection, embedding gather, the attention delta = rowsum(O*dO),
// cut-CE partial-statistics combine, sum of squares for the global gradient norm and the
// fused AdamW update with moments in the parameter dtype.
//
// All of them move 16 bytes per thread per access and keep reductions in fp32.
// Reference semantics: rms_norm (src/causal_trainer/modeling/architecture.py:155-162),
// apply_rotary_cos_sin (src/causal_trainer/modeling/rotary.py:132-204), _mlp_projection
// (architecture.py:205-229), optimizer update (src/causal_trainer/training/steps.py:172-186,
// src/causal_trainer/training/optimizer.py:42-75).
#include <cuda_bf16.h>

#include "attention.h"

namespace ctb {
namespace ew {

constexpr int NORM_THREADS = 256;
constexpr int NORM_MAXV = 8;  // 8-element vectors per thread: hidden size up to 16384

struct bf16x8 {
  uint4 raw;
};
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return raw;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sum over the block; every thread gets the result.  `scratch` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? scratch[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

// ------------------------------------------------------------------------------------------
// RMSNorm forward.  y = bf16(x * rstd) * w   (normalised value rounded to bf16 before the
// scale, as the reference does).  With `residual` set: h = x + residual is written to
// `h_out` first and normalised.
// ------------------------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual,
                   const __nv_bfloat16* w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, int rows, int d, float eps) {
  let_successor_start();
  wait_for_predecessor();
  __shared__ float scratch[33];
  const int nvec = d / 8;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * d);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * d) : nullptr;
    uint4 hv[NV];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * NORM_THREADS;
      if (v < nvec) {
        float f[8];
        unpack8(xr[v], f);
        if (rr) {
          float g[8];
          unpack8(rr[v], g);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __bfloat162float(__float2bfloat16(f[e] + g[e]));
          hv[i] = pack8(f);
          reinterpret_cast<uint4*>(h_out + static_cast<size_t>(row) * d)[v] = hv[i];
        } else {
          hv[i] = xr[v];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
      }
    }
    const float total = block_sum(ss, scratch);
    const float rstd = rsqrtf(total / d + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * NORM_THREADS;
      if (v < nvec) {
        float f[8], g[8];
        unpack8(hv[i], f);
        unpack8(reinterpret_cast<const uint4*>(w)[v], g);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __bfloat162float(__float2bfloat16(f[e] * rstd)) * g[e];
        reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * d)[v] = pack8(f);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// RMSNorm backward.  dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres), and per-CTA
// partial sums of dw = sum_rows dy * xhat into `dw_partial[gridDim.x][d]` (fp32 scratch),
// reduced by rmsnorm_dw_reduce_kernel.  No atomics: the result is deterministic.
// ------------------------------------------------------------------------------------------
// The loads of the next row are issued before the current row is reduced (d <= 4096: wider rows have no
// registers for it), and the row sum takes one barrier (two alternating sets of warp sums): with the loads, two
// barriers and the residual load in one chain per row, two CTAs per SM kept too little in flight.  16384 rows, us
// before and now: d = 4096 217 and 112; 8192, one CTA per SM for its 179 registers, 384 and 249; 16384 1297 and 832.
template <int NV>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                   const __nv_bfloat16* w, const float* rstd,
                   const __nv_bfloat16* dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, int rows, int d) {
  let_successor_start();
  wait_for_predecessor();
  constexpr int WARPS = NORM_THREADS / 32;
  constexpr bool AHEAD = NV <= 2;
  constexpr bool HOLD = NV <= 4;          // w and the residual gradient in registers (else read where they are used)
  __shared__ float sums[2][WARPS];
  const int nvec = d / 8;
  float dw_acc[NV][8];
  uint4 wv[NV], dyv[NV], xv[NV], rv[NV];
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * NORM_THREADS;
    if (HOLD) wv[i] = v < nvec ? reinterpret_cast<const uint4*>(w)[v] : zero;
    rv[i] = zero;
#pragma unroll
    for (int e = 0; e < 8; ++e) dw_acc[i][e] = 0.f;
  }
  float rs = 0.f;
  auto fetch = [&](int row) {
    const size_t at = static_cast<size_t>(row) * nvec;
    rs = rstd[row];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * NORM_THREADS;
      if (v < nvec) {
        dyv[i] = reinterpret_cast<const uint4*>(dy)[at + v];
        xv[i] = reinterpret_cast<const uint4*>(x)[at + v];
        if (HOLD && dres) rv[i] = reinterpret_cast<const uint4*>(dres)[at + v];
      } else {
        dyv[i] = xv[i] = zero;
      }
    }
  };
  if (AHEAD && blockIdx.x < rows) fetch(blockIdx.x);
  int parity = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, parity ^= 1) {
    if (!AHEAD) fetch(row);
    const float r_now = rs;
    uint4 dy_now[NV], x_now[NV], res_now[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      dy_now[i] = dyv[i];
      x_now[i] = xv[i];
      res_now[i] = rv[i];
    }
    if (AHEAD && row + static_cast<int>(gridDim.x) < rows) fetch(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float a[8], b[8], c[8];
      unpack8(dy_now[i], a);
      unpack8(x_now[i], b);
      const int v = threadIdx.x + i * NORM_THREADS;
      unpack8(HOLD ? wv[i] : (v < nvec ? reinterpret_cast<const uint4*>(w)[v] : zero), c);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xh = b[e] * r_now;
        dot += a[e] * c[e] * xh;
        dw_acc[i][e] += a[e] * xh;
      }
    }
    // (not held: w and the residual gradient are read two vectors ahead, because they could not pass the barrier and the stores)
    uint4 w_at[3], r_at[3];
    auto fetch_wide = [&](int i) {
      const int v = threadIdx.x + i * NORM_THREADS;
      r_at[i % 3] = zero;
      if (v < nvec) {
        w_at[i % 3] = reinterpret_cast<const uint4*>(w)[v];
        if (dres) r_at[i % 3] = reinterpret_cast<const uint4*>(dres)[static_cast<size_t>(row) * nvec + v];
      }
    };
    if (!HOLD) {
      fetch_wide(0);
      fetch_wide(1);
    }
    dot = warp_sum(dot);
    if ((threadIdx.x & 31) == 0) sums[parity][threadIdx.x >> 5] = dot;
    __syncthreads();
    float mean = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) mean += sums[parity][k];
    mean /= d;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * NORM_THREADS;
      if (!HOLD && i + 2 < NV) fetch_wide(i + 2);
      if (v < nvec) {
        float a[8], b[8], c[8], r[8], o[8];
        unpack8(dy_now[i], a);
        unpack8(x_now[i], b);
        unpack8(HOLD ? wv[i] : w_at[i % 3], c);
        unpack8(HOLD ? res_now[i] : r_at[i % 3], r);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = r_now * (a[e] * c[e] - b[e] * r_now * mean) + r[e];
        reinterpret_cast<uint4*>(dx + static_cast<size_t>(row) * d)[v] = pack8(o);
      }
    }
  }
  float* out = dw_partial + static_cast<size_t>(blockIdx.x) * d;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * NORM_THREADS;
    if (v < nvec) {
      float4* o4 = reinterpret_cast<float4*>(out + v * 8);
      o4[0] = make_float4(dw_acc[i][0], dw_acc[i][1], dw_acc[i][2], dw_acc[i][3]);
      o4[1] = make_float4(dw_acc[i][4], dw_acc[i][5], dw_acc[i][6], dw_acc[i][7]);
    }
  }
}

// dw[c] (+)= sum_p partial[p][c]; out dtype bf16 or fp32.  A block takes 32 columns, its warps take
// every DW_WARPS-th partial row (128 bytes a row) and join through shared memory in a fixed order.  Few blocks and all latency:
// with one thread per column walking all rows, the 16 blocks of d = 4096 were a chain of 296 loads; with 8 warps instead of
// 32 the whole backward norm of 512 x 256 takes 6.8 us for 4.8, of 1000 x 1536 9.1 for 7.3, of 8192 x 1536 29.0 for 27.0.
template <int DW_WARPS>
__global__ void __launch_bounds__(DW_WARPS * 32)
rmsnorm_dw_reduce_kernel(const float* partial, int parts, int d, void* __restrict__ dw, int out_f32,
                         int accumulate) {
  let_successor_start();
  wait_for_predecessor();
  __shared__ float sums[DW_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < d) {
#pragma unroll 8
    for (int p = warp; p < parts; p += DW_WARPS) s += partial[static_cast<size_t>(p) * d + c];
  }
  sums[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || c >= d) return;
#pragma unroll
  for (int k = 1; k < DW_WARPS; ++k) s += sums[k][lane];
  if (out_f32) {
    float* o = static_cast<float*>(dw);
    o[c] = accumulate ? o[c] + s : s;
  } else {
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(dw);
    o[c] = __float2bfloat16(accumulate ? __bfloat162float(o[c]) + s : s);
  }
}

// Column sums of a bf16 matrix (the gradient of a projection's bias) into per-CTA partial rows, which
// rmsnorm_dw_reduce_kernel adds up.  Bound by reading the matrix once: a warp reads 512 bytes of a row, eight
// rows a CTA, and the next four rows a warp are on their way while four are added (8192 x 2048 6.7 us; in a loop that the compiler
// unrolls by four 11.9, four at a time 10.2); the cast to fp32 and the strided sum that did this wrote and read
// twice the matrix in between.
__global__ void __launch_bounds__(256)
column_sum_kernel(const __nv_bfloat16* x, long ld, int rows, int n, float* __restrict__ partial) {
  let_successor_start();
  wait_for_predecessor();
  constexpr int AHEAD = 4;                       // rows; the loads of as many more are in flight behind them
  __shared__ float sums[8][256 + 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 256 + lane * 8;
  const bool live = c < n;
  const int step = gridDim.y * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (live) {
    uint4 raw[2][AHEAD];
    auto load = [&](int r, uint4 (&to)[AHEAD]) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        to[k] = make_uint4(0u, 0u, 0u, 0u);
        if (r + k * step < rows) to[k] = *reinterpret_cast<const uint4*>(x + static_cast<long>(r + k * step) * ld + c);
      }
    };
    auto add = [&](const uint4 (&from)[AHEAD]) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        float f[8];
        unpack8(from[k], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += f[e];
      }
    };
    int r = blockIdx.y * 8 + warp;
    load(r, raw[0]);
    while (r < rows) {
      load(r += AHEAD * step, raw[1]);
      add(raw[0]);
      load(r += AHEAD * step, raw[0]);
      add(raw[1]);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) sums[warp][e * 33 + lane] = acc[e];
  __syncthreads();
  // thread t: column t of the block's 256
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col >= n) return;
  const int at = (threadIdx.x & 7) * 33 + (threadIdx.x >> 3);
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) t += sums[w][at];
  partial[static_cast<size_t>(blockIdx.y) * n + col] = t;
}

// ------------------------------------------------------------------------------------------
// RoPE, in place on `heads` consecutive heads of a packed projection row.
//   x: [T][row_stride] with head h at columns h*D..h*D+D-1; cos/sin: [T][rot/2] fp32.
//   style 0 = gpt-j (adjacent pairs), 1 = gpt-neox (half split).  sign=-1 applies the
//   inverse rotation (the backward pass).
// ------------------------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* cosv,
                            const float* sinv, long row_stride, int T, int heads, int D, int rot,
                            int style, float sign) {
  let_successor_start();
  wait_for_predecessor();
  const int half = rot / 2;
  const long total = static_cast<long>(T) * heads * half;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(i % half);
    const long th = i / half;
    const int h = static_cast<int>(th % heads);
    const long t = th / heads;
    const float c = cosv[t * half + p];
    const float s = sinv[t * half + p] * sign;
    __nv_bfloat16* base = x + t * row_stride + static_cast<long>(h) * D;
    const int i0 = style == 0 ? 2 * p : p;
    const int i1 = style == 0 ? 2 * p + 1 : p + half;
    const float a = __bfloat162float(base[i0]);
    const float b = __bfloat162float(base[i1]);
    base[i0] = __float2bfloat16(a * c - b * s);
    base[i1] = __float2bfloat16(b * c + a * s);
  }
}

// The same on 16-byte vectors: a warp owns a token, a lane keeps the cos / sin of its channels in
// registers and walks the heads, so the table is read once per token instead of once per head and
// the projection moves in whole 128-byte segments.  Bound by reading and writing the rotated heads once.
// Where there are too few tokens to fill the GPU, 2^share warps share the heads of a token.
//   gpt-neox: a lane holds channels [8 p, 8 p + 8) of both halves;  gpt-j: four adjacent pairs.
template <int STYLE, bool SHARED>
__global__ void __launch_bounds__(256)
rope_vec_kernel(__nv_bfloat16* __restrict__ x, const float* cosv, const float* sinv,
                long row_stride, int T, int heads, int D, int rot, float sign, int share) {
  let_successor_start();
  wait_for_predecessor();
  constexpr int N = STYLE == 0 ? 4 : 8;          // angles per lane
  const int half = rot / 2;
  const int per_head = half / N;                 // lanes per head (<= 32)
  const int lane = threadIdx.x & 31;
  const int together = 32 / per_head;            // heads a warp rotates at once
  const int p = lane % per_head, first = lane / per_head;
  if (first >= together) return;
  if (!SHARED) share = 0;
  const long warps = ((static_cast<long>(gridDim.x) * blockDim.x) >> 5) >> share;
  const long warp = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int stride = together << share, h0 = first + (static_cast<int>(warp) & ((1 << share) - 1)) * together;
  for (long t = warp >> share; t < T; t += warps) {
    float c[N], s[N];
#pragma unroll
    for (int e = 0; e < N; e += 4) {
      *reinterpret_cast<float4*>(c + e) = *reinterpret_cast<const float4*>(cosv + t * half + p * N + e);
      *reinterpret_cast<float4*>(s + e) = *reinterpret_cast<const float4*>(sinv + t * half + p * N + e);
    }
#pragma unroll
    for (int e = 0; e < N; ++e) s[e] *= sign;
    __nv_bfloat16* row = x + t * row_stride + 8 * p;
#pragma unroll 4
    for (int h = h0; h < heads; h += stride) {
      uint4* at = reinterpret_cast<uint4*>(row + static_cast<long>(h) * D);
      float a[8], b[8], o[8];
      unpack8(at[0], a);
      if (STYLE == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o[2 * e] = a[2 * e] * c[e] - a[2 * e + 1] * s[e];
          o[2 * e + 1] = a[2 * e + 1] * c[e] + a[2 * e] * s[e];
        }
      } else {
        uint4* up = reinterpret_cast<uint4*>(row + static_cast<long>(h) * D + half);
        unpack8(up[0], b);
        float q[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          o[e] = a[e] * c[e] - b[e] * s[e];
          q[e] = b[e] * c[e] + a[e] * s[e];
        }
        up[0] = pack8(q);
      }
      at[0] = pack8(o);
    }
  }
}

// cos/sin tables from arbitrary integer positions: angle = pos * inv_freq[p] in fp32.
__global__ void rope_table_kernel(const int* __restrict__ pos, const float* __restrict__ inv_freq,
                                  float* __restrict__ cosv, float* __restrict__ sinv, int T, int half) {
  const long total = static_cast<long>(T) * half;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(i % half);
    const long t = i / half;
    const float ang = static_cast<float>(pos[t]) * inv_freq[p];
    float s, c;
    sincosf(ang, &s, &c);
    // the reference casts the table to the compute dtype once per step
    cosv[i] = __bfloat162float(__float2bfloat16(c));
    sinv[i] = __bfloat162float(__float2bfloat16(s));
  }
}

// ------------------------------------------------------------------------------------------
// SwiGLU on the packed projection gu[T][2f] = [gate | up]:  h = silu(gate) * up.
// Backward writes d(gate|up) in the same packed layout.
// ------------------------------------------------------------------------------------------
// n / d for d = 1 + exp(-g), g below 87 in size, and |n| <= 87, by Markstein's method (P. W. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990): a reciprocal refined by a Newton step, a quotient
// of it, and that quotient corrected by its remainder.  Why it holds here: 1 <= d < 2^126, so that the reciprocal is a normal
// number; after the step it is within half an ulp and a little of 1 / d (the approximate one is within 2^-23, the step squares that), the
// quotient within an ulp of n / d, and the remainder of such a quotient is a number that the fused multiply-add gives exactly.  The sum
// before its one rounding is within 2^-46 of n / d, so only a quotient that close to the middle of two fp32 numbers could come out as the
// other one.  tests/test_kernel_edges_gpu.py compares all gates of bf16 with the division: no result differs.
// The division bound the forward kernel by its instructions (280 us at 16384 x 14336, so 234); a fast one returns zero for
// denominators above 2^126, gates between -88.7 and -87.4.  A vector with a larger gate, or one that is not a number, divides, in a
// function of its own: inlined it costs the others their registers (260 us).
__device__ __forceinline__ float quotient_in_range(float n, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-d, r, 1.f), r);
  const float q = n * r;
  return fmaf(fmaf(-q, d, n), r, q);
}
// Whether the eight gates of every lane that has come here are below 87 (0x42ae) in size, as bf16 bit patterns.  One answer for the
// warp: with lanes apart it runs both quotients one after the other (1000 x 8960 in a sequence, gates of size 39, forward and
// backward: 23.4 and 24.1 us, where the division alone took 16.8 and 17.7; so 1.04 and 1.09 of the division's time, of gates of size 20
// 0.81 and 0.95).
__device__ __forceinline__ bool gates_in_range(const uint4& gates) {
  const unsigned m = __vmaxu2(__vmaxu2(gates.x & 0x7fff7fffu, gates.y & 0x7fff7fffu),
                              __vmaxu2(gates.z & 0x7fff7fffu, gates.w & 0x7fff7fffu));
  return __all_sync(__activemask(), (m & 0xffffu) < 0x42aeu && (m >> 16) < 0x42aeu);
}
template <bool PLAIN>
__device__ __forceinline__ uint4 swiglu_vector(const uint4& gates, const uint4& ups) {
  float g[8], u[8], o[8];
  unpack8(gates, g);
  unpack8(ups, u);
  const unsigned words[4] = {gates.x, gates.y, gates.z, gates.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float d0 = 1.f + __expf(-g[2 * i]), d1 = 1.f + __expf(-g[2 * i + 1]);
    __nv_bfloat162 act = PLAIN ? __floats2bfloat162_rn(quotient_in_range(g[2 * i], d0), quotient_in_range(g[2 * i + 1], d1))
                               : __floats2bfloat162_rn(g[2 * i] / d0, g[2 * i + 1] / d1);
    // (the corrected quotient of -0 is +0)
    if (PLAIN) *reinterpret_cast<unsigned*>(&act) |= words[i] & 0x80008000u;
    const float2 a = __bfloat1622float2(act);
    o[2 * i] = a.x * u[2 * i];
    o[2 * i + 1] = a.y * u[2 * i + 1];
  }
  return pack8(o);
}
struct GateUp {
  uint4 gate, up;
};
template <bool PLAIN>
__device__ __forceinline__ GateUp swiglu_gradient(const uint4& gates, const uint4& ups, const uint4& grads) {
  float g[8], u[8], d[8], dg[8], du[8];
  unpack8(gates, g);
  unpack8(ups, u);
  unpack8(grads, d);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float den = 1.f + __expf(-g[e]);
    const float sg = PLAIN ? quotient_in_range(1.f, den) : 1.f / den;
    const float act = g[e] * sg;
    du[e] = d[e] * act;
    dg[e] = d[e] * u[e] * sg * (1.f + g[e] * (1.f - sg));
  }
  return {pack8(dg), pack8(du)};
}
__device__ __noinline__ uint4 swiglu_vector_of_any(uint4 gates, uint4 ups) { return swiglu_vector<false>(gates, ups); }
__device__ __noinline__ GateUp swiglu_gradient_of_any(uint4 gates, uint4 ups, uint4 grads) {
  return swiglu_gradient<false>(gates, ups, grads);
}

// A thread takes every gridDim * blockDim-th 16-byte vector of h and steps its row along instead of dividing for
// it, so no thread idles whatever the width (a column per thread and rows over blockIdx.y left 224 of 256 idle at
// f = 256: 100000 x 256 82 us forward where this takes 36).  The forward kernel keeps two vectors in flight where
// a thread has ten or more, the backward kernel one.  Both are bound by memory; the grids are chosen where they are launched.
struct SwigluWalk {
  long i, total, stride;      // vector of h; number of them; step
  long row_at, row_step;      // (row of i) * nvec: the gate vector of i is i + row_at, its up vector nvec further
  int v, v_step, nvec;        // column of i
  __device__ __forceinline__ SwigluWalk(long T, int f) {
    nvec = f / 8;
    total = T * nvec;
    const unsigned first = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;   // (a few hundred thousand)
    i = first;
    stride = all;
    v = static_cast<int>(first % nvec);
    row_at = i - v;
    v_step = static_cast<int>(all % nvec);
    row_step = stride - v_step;
  }
  __device__ __forceinline__ void step() {
    i += stride;
    v += v_step;
    row_at += row_step;
    if (v >= nvec) {
      v -= nvec;
      row_at += nvec;
    }
  }
};
template <int AHEAD>      // vectors in flight
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* __restrict__ h, long T, int f) {
  let_successor_start();
  wait_for_predecessor();
  const uint4* src = reinterpret_cast<const uint4*>(gu);
  SwigluWalk w(T, f);
  while (w.i < w.total) {
    uint4 gv[AHEAD], uv[AHEAD];
    long to[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      to[k] = w.i;
      if (w.i < w.total) {
        gv[k] = src[w.i + w.row_at];
        uv[k] = src[w.i + w.row_at + w.nvec];
      }
      w.step();
    }
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
      if (to[k] < w.total) {
        reinterpret_cast<uint4*>(h)[to[k]] =
            gates_in_range(gv[k]) ? swiglu_vector<true>(gv[k], uv[k]) : swiglu_vector_of_any(gv[k], uv[k]);
      }
  }
}
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* dh,
                  __nv_bfloat16* __restrict__ dgu, long T, int f) {
  let_successor_start();
  wait_for_predecessor();
  const uint4* src = reinterpret_cast<const uint4*>(gu);
  uint4* dst = reinterpret_cast<uint4*>(dgu);
  for (SwigluWalk w(T, f); w.i < w.total; w.step()) {
    const long at = w.i + w.row_at;
    const uint4 gv = src[at], uv = src[at + w.nvec], dv = reinterpret_cast<const uint4*>(dh)[w.i];
    const GateUp r = gates_in_range(gv) ? swiglu_gradient<true>(gv, uv, dv) : swiglu_gradient_of_any(gv, uv, dv);
    dst[at] = r.gate;
    dst[at + w.nvec] = r.up;
  }
}

// ------------------------------------------------------------------------------------------
// Embedding gather: out[t] = table[ids[t]] (the stored pad row is returned as is).
// ------------------------------------------------------------------------------------------
__global__ void embedding_gather_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                        __nv_bfloat16* __restrict__ out, long T, int d, int vocab) {
  const int nvec = d / 8;
  const long total = T * nvec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long t = i / nvec;
    const int v = static_cast<int>(i % nvec);
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    reinterpret_cast<uint4*>(out + t * d)[v] = reinterpret_cast<const uint4*>(table + static_cast<long>(id) * d)[v];
  }
}

// ------------------------------------------------------------------------------------------
// delta[b][h][s] = sum_d O[b][s][h][d] * dO[b][s][h][d]   (one warp per (token, head))
// ------------------------------------------------------------------------------------------
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                  float* __restrict__ delta, int B, int S, int H, int D, long o_rs, long do_rs) {
  const long warp_id = (blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long total = static_cast<long>(B) * S * H;
  if (warp_id >= total) return;
  const int h = static_cast<int>(warp_id % H);
  const long t = warp_id / H;
  const __nv_bfloat16* op = o + t * o_rs + static_cast<long>(h) * D;
  const __nv_bfloat16* dp = dout + t * do_rs + static_cast<long>(h) * D;
  float acc = 0.f;
  for (int c = lane * 2; c < D; c += 64) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(op + c));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dp + c));
    acc += a.x * b.x + a.y * b.y;
  }
  acc = warp_sum(acc);
  if (lane == 0) {
    const long b_idx = t / S, s_idx = t % S;
    delta[(b_idx * H + h) * S + s_idx] = acc;
  }
}

// ------------------------------------------------------------------------------------------
// Per-query statistics of the attention backward, in the form its kernels consume:
//   neg_delta[b][h][s] = -sum_d O dO        neg_lse2[b][h][s] = -lse[b][h][s] * log2(e)
// (one warp per (token, head)), so the inner loops use packed fma / add without a negation.
// ------------------------------------------------------------------------------------------
__global__ void attn_bwd_stats_kernel(const __nv_bfloat16* o, const __nv_bfloat16* dout,
                                      const float* lse, float* __restrict__ neg_lse2,
                                      float* __restrict__ neg_delta, int B, int S, int H, int D, long o_rs, long do_rs) {
  let_successor_start();
  wait_for_predecessor();
  const long warp_id = (blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long total = static_cast<long>(B) * S * H;
  if (warp_id >= total) return;
  const int h = static_cast<int>(warp_id % H);
  const long t = warp_id / H;
  const __nv_bfloat16* op = o + t * o_rs + static_cast<long>(h) * D;
  const __nv_bfloat16* dp = dout + t * do_rs + static_cast<long>(h) * D;
  float acc = 0.f;
  for (int c = lane * 2; c < D; c += 64) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(op + c));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dp + c));
    acc += a.x * b.x + a.y * b.y;
  }
  acc = warp_sum(acc);
  if (lane == 0) {
    const long b_idx = t / S, s_idx = t % S;
    const long i = (b_idx * H + h) * S + s_idx;
    neg_delta[i] = -acc;
    neg_lse2[i] = -lse[i] * 1.4426950408889634f;
  }
}

// The same for D = 64 or 128 and 16-byte aligned rows.  Bound by reading O and dO once.  The kernel
// above reads 4 bytes per lane and access and stores one float per warp, S floats apart; here a
// group of D / 8 lanes reads a (token, head) row as 16-byte vectors, a block takes STAT_TOKENS tokens
// x STAT_HEADS heads (1 KiB contiguous per token at D = 128) and turns the sums round in shared memory, so that
// lse is read and both statistics are written 128 bytes at a time.  With 8 heads a block (us; 4 heads behind it): 8 rows of 4096 tokens,
// 12 heads 43.8, 37.5; 1 of 4096, 28 heads 9.9, 8.3; 4 of 1024, 32 heads 10.0, 9.1; 1 of 32768, 8 heads 27.3, 28.3.
// The loads of four passes are issued before the sums of the first: left to the compiler, which may not move ordinary loads over the
// stores of the sums, 1 of 4096, 28 heads took 11.5.
constexpr int STAT_TOKENS = 32, STAT_HEADS = 4;
template <int D>
__global__ void __launch_bounds__(256)
attn_bwd_stats_vec_kernel(const __nv_bfloat16* o, const __nv_bfloat16* dout,
                          const float* lse, float* __restrict__ neg_lse2,
                          float* __restrict__ neg_delta, int S, int H, long tokens, long o_rs, long do_rs) {
  let_successor_start();
  wait_for_predecessor();
  constexpr int LANES = D / 8;                   // lanes per (token, head) row
  constexpr int ROWS = 256 / LANES;              // rows per pass of the block
  constexpr int PASSES = STAT_TOKENS * STAT_HEADS / ROWS;
  __shared__ float sums[STAT_HEADS][STAT_TOKENS + 1];
  const long t0 = static_cast<long>(blockIdx.x) * STAT_TOKENS;
  const int h0 = blockIdx.y * STAT_HEADS;
  const int sub = threadIdx.x / LANES, c = (threadIdx.x % LANES) * 8;
  constexpr int AHEAD = 4;
  static_assert(PASSES % AHEAD == 0, "whole groups of passes");
  for (int p0 = 0; p0 < PASSES; p0 += AHEAD) {
    uint4 av[AHEAD], bv[AHEAD];
#pragma unroll
    for (int p = 0; p < AHEAD; ++p) {
      const int row = (p0 + p) * ROWS + sub, hl = row % STAT_HEADS, tl = row / STAT_HEADS;
      av[p] = bv[p] = make_uint4(0u, 0u, 0u, 0u);
      if (t0 + tl < tokens && h0 + hl < H) {
        const long at = static_cast<long>(h0 + hl) * D + c;
        av[p] = *reinterpret_cast<const uint4*>(o + (t0 + tl) * o_rs + at);
        bv[p] = *reinterpret_cast<const uint4*>(dout + (t0 + tl) * do_rs + at);
      }
    }
#pragma unroll
    for (int p = 0; p < AHEAD; ++p) {
      const int row = (p0 + p) * ROWS + sub;
      float a[8], b[8], acc = 0.f;
      unpack8(av[p], a);
      unpack8(bv[p], b);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += a[e] * b[e];
#pragma unroll
      for (int m = LANES / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
      if (c == 0) sums[row % STAT_HEADS][row / STAT_HEADS] = acc;
    }
  }
  __syncthreads();
  const int hl = threadIdx.x >> 5, tl = threadIdx.x & 31;
  const long t = t0 + tl;
  if (hl >= STAT_HEADS || t >= tokens || h0 + hl >= H) return;
  const long i = (t / S * H + h0 + hl) * S + t % S;
  neg_delta[i] = -sums[hl][tl];
  neg_lse2[i] = -lse[i] * 1.4426950408889634f;
}

// ------------------------------------------------------------------------------------------
// Cut-CE combine: merges per-slab (max, sumexp) into lse[row], emits the weighted NLL per
// row, the backward coefficient coef[row] = weight * grad_scale, and block partial sums of
// (nll, weight) which the host-side wrapper adds up (fp32, fixed order: deterministic).
// ------------------------------------------------------------------------------------------
// A block takes CE_ROWS rows (one per lane); its warps share the slabs and join through shared memory in a
// fixed order.  With a thread walking all slabs of its row, the 16 blocks of 4096 rows were a chain of
// 2 x 501 loads (129 us).
constexpr int CE_ROWS = 32, CE_WARPS = 8;
__global__ void __launch_bounds__(CE_ROWS * CE_WARPS)
ce_combine_kernel(const float* pmax, const float* psum, int slabs,
                  const float* target_logit, const int* targets, int target_step, int vocab,
                  const float* weights, float grad_scale, const float* scale,
                  float* __restrict__ lse, float* __restrict__ coef, float* __restrict__ block_nll,
                  float* __restrict__ block_w, int rows) {
  let_successor_start();
  wait_for_predecessor();
  __shared__ float part[CE_WARPS][CE_ROWS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * CE_ROWS + lane;
  const bool live = row < rows;
  float m = -INFINITY;
  if (live) {
#pragma unroll 8
    for (int s = warp; s < slabs; s += CE_WARPS) m = fmaxf(m, pmax[static_cast<size_t>(s) * rows + row]);
  }
  part[warp][lane] = m;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < CE_WARPS; ++k) m = fmaxf(m, part[k][lane]);
  float acc = 0.f;
  if (live) {
#pragma unroll 8
    for (int s = warp; s < slabs; s += CE_WARPS) {
      const size_t i = static_cast<size_t>(s) * rows + row;
      acc += psum[i] * __expf(pmax[i] - m);
    }
  }
  __syncthreads();
  part[warp][lane] = acc;
  __syncthreads();
  if (warp != 0) return;
  acc = 0.f;
#pragma unroll
  for (int k = 0; k < CE_WARPS; ++k) acc += part[k][lane];
  float nll = 0.f, w = 0.f;
  if (live) {
    const float l = m + logf(acc);
    lse[row] = l;
    w = weights[row];
    coef[row] = w * grad_scale * (scale != nullptr ? *scale : 1.f);
    // (the statistics write the logit of a target that is in the vocabulary, and nothing else)
    const int t = targets[static_cast<long>(row) * target_step];
    nll = (w != 0.f) ? (l - (t >= 0 && t < vocab ? target_logit[row] : 0.f)) * w : 0.f;
  }
  nll = warp_sum(nll);
  w = warp_sum(w);
  if (lane == 0) {
    block_nll[blockIdx.x] = nll;
    block_w[blockIdx.x] = w;
  }
}

// Sums of the blocks' partial sums, in a fixed order: one block, both sums (two reductions of the framework took 3.5 us each and
// a launch gap, this 2 behind the combine that it is chained to).
__global__ void __launch_bounds__(256)
ce_sums_kernel(const float* block_nll, const float* block_w, int blocks, float* __restrict__ nll,
               float* __restrict__ w) {
  let_successor_start();
  wait_for_predecessor();
  __shared__ float scratch[33];
  float a = 0.f, b = 0.f;
  for (int i = threadIdx.x; i < blocks; i += 256) {
    a += block_nll[i];
    b += block_w[i];
  }
  a = block_sum(a, scratch);
  b = block_sum(b, scratch);
  if (threadIdx.x == 0) {
    *nll = a;
    *w = b;
  }
}

// ------------------------------------------------------------------------------------------
// Cross-entropy over a materialised logits slab [rows, vocab] (bf16): one CTA per row.
//   stats:    lse[row] = logsumexp(logits[row, :]), target_logit[row] (0 when the target is < 0)
//   backward: logits[row, v] <- (exp(logits[row, v] - lse[row]) - [v == target]) * coef[row], in place
// The projection-fused cut cross-entropy never writes logits; these two kernels are the variant
// that does (the reference's `pallas` loss backend, src/causal_trainer/kernels/cross_entropy.py:
// 99-189, 254-322), for when the slab is wanted anyway.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
logits_ce_stats_kernel(const __nv_bfloat16* __restrict__ logits, long ld, int vocab, const int* __restrict__ targets,
                       float* __restrict__ lse, float* __restrict__ target_logit) {
  __shared__ float scratch[33];
  __shared__ float s_max;
  const long row = blockIdx.x;
  const __nv_bfloat16* x = logits + row * ld;
  const int nvec = vocab / 8;
  float m = -INFINITY;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 raw = reinterpret_cast<const uint4*>(x)[v];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      m = fmaxf(m, fmaxf(f.x, f.y));
    }
  }
  for (int c = nvec * 8 + threadIdx.x; c < vocab; c += blockDim.x) m = fmaxf(m, __bfloat162float(x[c]));
  // block max through the sum helper's scratch: reduce per warp, then across warps
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = -INFINITY;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t = fmaxf(t, scratch[w]);
    s_max = t;
  }
  __syncthreads();
  const float mx = s_max;
  float acc = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 raw = reinterpret_cast<const uint4*>(x)[v];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      acc += __expf(f.x - mx) + __expf(f.y - mx);
    }
  }
  for (int c = nvec * 8 + threadIdx.x; c < vocab; c += blockDim.x) acc += __expf(__bfloat162float(x[c]) - mx);
  const float total = block_sum(acc, scratch);
  if (threadIdx.x == 0) {
    lse[row] = mx + logf(total);
    const int t = targets[row];
    target_logit[row] = (t >= 0 && t < vocab) ? __bfloat162float(x[t]) : 0.f;
  }
}

__global__ void __launch_bounds__(256)
logits_ce_backward_kernel(__nv_bfloat16* __restrict__ logits, long ld, int vocab, const int* __restrict__ targets,
                          const float* __restrict__ lse, const float* __restrict__ coef) {
  const long row = blockIdx.x;
  __nv_bfloat16* x = logits + row * ld;
  const float l = lse[row], c = coef[row];
  const int t = targets[row];
  const int nvec = vocab / 8;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    uint4 raw = reinterpret_cast<uint4*>(x)[v];
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      const int col = v * 8 + e * 2;
      const float a = (__expf(f.x - l) - (col == t ? 1.f : 0.f)) * c;
      const float b = (__expf(f.y - l) - (col + 1 == t ? 1.f : 0.f)) * c;
      h[e] = __floats2bfloat162_rn(a, b);
    }
    reinterpret_cast<uint4*>(x)[v] = raw;
  }
  for (int col = nvec * 8 + threadIdx.x; col < vocab; col += blockDim.x)
    x[col] = __float2bfloat16((__expf(__bfloat162float(x[col]) - l) - (col == t ? 1.f : 0.f)) * c);
}

// ------------------------------------------------------------------------------------------
// Gradients of kept fp32 logits, bf16, in the place of the logits: row r of the gradient begins where row r of the logits
// does.  A block walks a row in chunks; chunk k is written over logits that chunk k / 2 held, which every thread has read
// when it has passed the barrier of chunk k.  The expression is the one of the GEMM epilogue that recomputes the logits.
// Bound by memory: 6 bytes an element.
// Not chained to the launch before it (launch_chained), though the launch behind it may be: its blocks, a row each, would
// start while the product that writes the logits holds most SMs and crowd on those that it leaves first.  The whole loss of
// 100, 256 and 333 rows, 32000 x 1536, us, chained and not: 117, 146, 176 and 106, 133, 169; as a graph 113, 141, 167 and 101, 123, 159.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
kept_logits_gradient_kernel(float* __restrict__ logits, long ld, int vocab, const int* __restrict__ targets, int target_step,
                            const float* __restrict__ lse, const float* __restrict__ coef) {
  let_successor_start();
  const long row = blockIdx.x;
  const float* x = logits + row * ld;
  __nv_bfloat16* g = reinterpret_cast<__nv_bfloat16*>(logits + row * ld);
  const float l = lse[row], c = coef[row];
  const int t = targets[row * target_step];
  const int chunks = (vocab + 2047) / 2048;
  float4 a[2], next[2] = {};
  auto load = [&](int k, float4 (&to)[2]) {
    const int col = k * 2048 + threadIdx.x * 8;
    if (col < vocab) {
      to[0] = __ldcs(reinterpret_cast<const float4*>(x + col));
      to[1] = __ldcs(reinterpret_cast<const float4*>(x + col) + 1);
    }
  };
  load(0, next);
  for (int k = 0; k < chunks; ++k) {
    a[0] = next[0];
    a[1] = next[1];
    if (k + 1 < chunks) load(k + 1, next);
    const int col = k * 2048 + threadIdx.x * 8;
    float v[8] = {a[0].x, a[0].y, a[0].z, a[0].w, a[1].x, a[1].y, a[1].z, a[1].w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float pv = __expf(v[e] - l);
      if (col + e == t) pv -= 1.f;
      v[e] = pv * c;
    }
    __syncthreads();
    if (col < vocab)
      *reinterpret_cast<uint4*>(g + col) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                                                      pack_bf16(v[6], v[7]));
  }
}

// ------------------------------------------------------------------------------------------
// Sum of squares (fp32) of a bf16 / fp32 vector into per-block partials.
// ------------------------------------------------------------------------------------------
// 16-byte loads, four in flight per thread (with one element per load: 3.0 TB/s on 872 MB of fp32); a
// vector whose base is not 16-byte aligned is read element by element.
__device__ __forceinline__ float square_of(float v, int round_bf16) {
  if (round_bf16) v = __bfloat162float(__float2bfloat16(v));
  return v * v;
}
template <typename T>
__global__ void __launch_bounds__(256)
sumsq_kernel(const T* __restrict__ x, long n, float* __restrict__ partial, int round_bf16) {
  constexpr int N = 16 / sizeof(T), UNROLL = 4;
  __shared__ float scratch[33];
  const long first = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  float acc = 0.f;
  auto add = [&](const uint4& raw) {
    if (sizeof(T) == 4) {
      acc += square_of(__uint_as_float(raw.x), round_bf16);
      acc += square_of(__uint_as_float(raw.y), round_bf16);
      acc += square_of(__uint_as_float(raw.z), round_bf16);
      acc += square_of(__uint_as_float(raw.w), round_bf16);
    } else {
      float f[8];
      unpack8(raw, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += f[e] * f[e];
    }
  };
  const long nvec = reinterpret_cast<uintptr_t>(x) % 16 == 0 ? n / N : 0;
  const uint4* xv = reinterpret_cast<const uint4*>(x);
  long i = first;
  for (; i + (UNROLL - 1) * stride < nvec; i += UNROLL * stride) {
    uint4 raw[UNROLL];
#pragma unroll
    for (int k = 0; k < UNROLL; ++k) raw[k] = __ldg(xv + i + k * stride);
#pragma unroll
    for (int k = 0; k < UNROLL; ++k) add(raw[k]);
  }
  for (; i < nvec; i += stride) add(__ldg(xv + i));
  for (long j = nvec * N + first; j < n; j += stride) acc += square_of(static_cast<float>(x[j]), round_bf16);
  const float t = block_sum(acc, scratch);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// ------------------------------------------------------------------------------------------
// Fused AdamW on a flat shard.  Moments are stored in the parameter dtype; the arithmetic is
// fp32.  `clip` points at a device scalar (global-norm clip coefficient, <= 1) so the
// optimizer never waits for the host; `decay` is 0 for vectors (norm scales, biases).
//   g' = g*clip; m = b1 m + (1-b1) g'; v = b2 v + (1-b2) g'^2
//   p += bf16( -lr * ( m/(1-b1^t) / (sqrt(v/(1-b2^t)) + eps) + decay * p ) )
// ------------------------------------------------------------------------------------------
template <typename GT>
__global__ void adamw_kernel(__nv_bfloat16* __restrict__ p, const GT* __restrict__ g, __nv_bfloat16* __restrict__ m,
                             __nv_bfloat16* __restrict__ v, long n, float lr, float b1, float b2, float eps,
                             float decay, float bc1, float bc2, const float* __restrict__ clip, float gscale,
                             int round_bf16) {
  const float cs = (clip ? *clip : 1.f) * gscale;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    float graw = static_cast<float>(g[i]);
    if (round_bf16) graw = __bfloat162float(__float2bfloat16(graw));
    const float gi = graw * cs;
    const float mi = b1 * __bfloat162float(m[i]) + (1.f - b1) * gi;
    const float vi = b2 * __bfloat162float(v[i]) + (1.f - b2) * gi * gi;
    const float pi = __bfloat162float(p[i]);
    const float upd = -lr * ((mi / bc1) / (sqrtf(vi / bc2) + eps) + decay * pi);
    m[i] = __float2bfloat16(mi);
    v[i] = __float2bfloat16(vi);
    p[i] = __float2bfloat16(pi + __bfloat162float(__float2bfloat16(upd)));
  }
}

// ------------------------------------------------------------------------------------------
// AdamW over a whole flat arena in one launch.  The arena is a sequence of regions
// [bounds[r], bounds[r+1]) with a mode each: 1 = weight decay, 0 = no decay, -1 = frozen (the
// region is skipped: no update, moments untouched).  16-byte accesses: eight elements of the
// parameter, both moments and the gradient per thread per round, two rounds in flight.
// ------------------------------------------------------------------------------------------
constexpr int ADAM_MAX_REGIONS = 512;

__device__ __forceinline__ float fast_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename GT>
__global__ void __launch_bounds__(256)
adamw_regions_kernel(__nv_bfloat16* __restrict__ p, const GT* __restrict__ g, __nv_bfloat16* __restrict__ m,
                     __nv_bfloat16* __restrict__ v, long n, const long* __restrict__ bounds,
                     const int* __restrict__ modes, int nreg, float lr, float b1, float b2, float eps, float decay,
                     float bc1, float bc2, const float* __restrict__ clip, float gscale, int round_bf16) {
  __shared__ long sb[ADAM_MAX_REGIONS + 1];
  __shared__ int sm[ADAM_MAX_REGIONS];
  for (int i = threadIdx.x; i <= nreg; i += blockDim.x) sb[i] = bounds[i];
  for (int i = threadIdx.x; i < nreg; i += blockDim.x) sm[i] = modes[i];
  __syncthreads();
  const float cs = (clip ? *clip : 1.f) * gscale;
  const float inv_bc1 = 1.f / bc1, inv_bc2 = 1.f / bc2;
  auto region_of = [&](long e) {
    int lo = 0, hi = nreg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sb[mid] <= e) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  const long nvec = n / 8;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  int cached = 0;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nvec; i += stride) {
    const long e0 = i * 8;
    if (!(sb[cached] <= e0 && e0 < sb[cached + 1])) cached = region_of(e0);
    const bool uniform = sb[cached + 1] >= e0 + 8;
    if (uniform && sm[cached] < 0) continue;
    uint4 pr = reinterpret_cast<const uint4*>(p)[i];
    uint4 mr = reinterpret_cast<const uint4*>(m)[i];
    uint4 vr = reinterpret_cast<const uint4*>(v)[i];
    float gf[8];
    if constexpr (sizeof(GT) == 4) {
      const float4 g0 = reinterpret_cast<const float4*>(g)[2 * i];
      const float4 g1 = reinterpret_cast<const float4*>(g)[2 * i + 1];
      gf[0] = g0.x; gf[1] = g0.y; gf[2] = g0.z; gf[3] = g0.w;
      gf[4] = g1.x; gf[5] = g1.y; gf[6] = g1.z; gf[7] = g1.w;
      if (round_bf16) {
#pragma unroll
        for (int e = 0; e < 8; ++e) gf[e] = __bfloat162float(__float2bfloat16(gf[e]));
      }
    } else {
      const uint4 gr = reinterpret_cast<const uint4*>(g)[i];
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gr);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(gh[e]);
        gf[2 * e] = f.x;
        gf[2 * e + 1] = f.y;
      }
    }
    __nv_bfloat16* pe = reinterpret_cast<__nv_bfloat16*>(&pr);
    __nv_bfloat16* me = reinterpret_cast<__nv_bfloat16*>(&mr);
    __nv_bfloat16* ve = reinterpret_cast<__nv_bfloat16*>(&vr);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int mode = uniform ? sm[cached] : sm[region_of(e0 + e)];
      if (mode < 0) continue;
      const float gi = gf[e] * cs;
      const float mi = b1 * __bfloat162float(me[e]) + (1.f - b1) * gi;
      const float vi = b2 * __bfloat162float(ve[e]) + (1.f - b2) * gi * gi;
      const float pi = __bfloat162float(pe[e]);
      // one sqrt.approx and one rcp.approx per element (2 ulp each, far below the bf16 rounding of the
      // update): with IEEE division and square root the sweep is bound by instruction issue, not by HBM
      const float upd = -lr * ((mi * inv_bc1) * fast_rcp(fast_sqrt(vi * inv_bc2) + eps) + (mode ? decay : 0.f) * pi);
      me[e] = __float2bfloat16(mi);
      ve[e] = __float2bfloat16(vi);
      pe[e] = __float2bfloat16(pi + __bfloat162float(__float2bfloat16(upd)));
    }
    reinterpret_cast<uint4*>(p)[i] = pr;
    reinterpret_cast<uint4*>(m)[i] = mr;
    reinterpret_cast<uint4*>(v)[i] = vr;
  }
}

// ------------------------------------------------------------------------------------------
// Active-row compaction (rows whose loss weight is non-zero go through the LM head; the others do
// not).  Stable: the compacted order is the row order, so results do not depend on it.
//   active_count   rows with weight != 0 per block of 1024 rows
//   active_fill    idx[k] = k-th active row; total[0] = number of active rows
//   gather_rows    dst[j] = src[idx[j]]
//   scatter_rows   dst[idx[j]] = src[j] for j < total (dst cleared by the caller)
// ------------------------------------------------------------------------------------------
constexpr int ACTIVE_BLOCK = 1024;

__global__ void __launch_bounds__(ACTIVE_BLOCK)
active_count_kernel(const float* __restrict__ w, int rows, int* __restrict__ block_counts) {
  const int r = blockIdx.x * ACTIVE_BLOCK + threadIdx.x;
  const int flag = (r < rows && w[r] != 0.f) ? 1 : 0;
  const int n = __syncthreads_count(flag);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = n;
}

__global__ void __launch_bounds__(ACTIVE_BLOCK)
active_fill_kernel(const float* __restrict__ w, int rows, const int* __restrict__ block_counts, int* __restrict__ idx,
                   int* __restrict__ total) {
  __shared__ int warp_sums[ACTIVE_BLOCK / 32];
  __shared__ int base_s;
  const int r = blockIdx.x * ACTIVE_BLOCK + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool flag = r < rows && w[r] != 0.f;
  const unsigned votes = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) warp_sums[warp] = __popc(votes);
  if (threadIdx.x == 0) {
    int base = 0;
    for (int b = 0; b < static_cast<int>(blockIdx.x); ++b) base += block_counts[b];
    base_s = base;
  }
  __syncthreads();
  int before = base_s;
  for (int x = 0; x < warp; ++x) before += warp_sums[x];
  if (flag) idx[before + __popc(votes & ((1u << lane) - 1u))] = r;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    int sum = base_s;
    for (int x = 0; x < ACTIVE_BLOCK / 32; ++x) sum += warp_sums[x];
    total[0] = sum;
  }
}

// Row indices come from device memory: an index outside [0, rows) is recorded in the status word
// (site, position, value) and the row is skipped; nothing is read or written out of bounds.
enum : unsigned { SITE_GATHER_INDEX = 0x0601, SITE_SCATTER_INDEX = 0x0602 };

__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ src, long src_stride, const int* __restrict__ idx,
                                   __nv_bfloat16* __restrict__ dst, long n, int d, int rows, DeviceStatus* st) {
  const int nvec = d / 8;
  const long work = n * nvec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < work;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long j = i / nvec;
    const int v = static_cast<int>(i % nvec);
    const int r = idx[j];
    if (r < 0 || r >= rows) {
      if (v == 0) report_failure(st, SITE_GATHER_INDEX, static_cast<unsigned>(j), static_cast<unsigned>(r));
      reinterpret_cast<uint4*>(dst + j * d)[v] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    reinterpret_cast<uint4*>(dst + j * d)[v] = reinterpret_cast<const uint4*>(src + r * src_stride)[v];
  }
}

__global__ void scatter_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ idx,
                                    const int* __restrict__ total, __nv_bfloat16* __restrict__ dst, long dst_stride,
                                    long n, int d, int rows, DeviceStatus* st) {
  const int nvec = d / 8;
  const long live = min(n, static_cast<long>(total[0]));
  const long work = live * nvec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < work;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long j = i / nvec;
    const int v = static_cast<int>(i % nvec);
    const int r = idx[j];
    if (r < 0 || r >= rows) {
      if (v == 0) report_failure(st, SITE_SCATTER_INDEX, static_cast<unsigned>(j), static_cast<unsigned>(r));
      continue;
    }
    reinterpret_cast<uint4*>(dst + r * dst_stride)[v] = reinterpret_cast<const uint4*>(src + j * d)[v];
  }
}

// ------------------------------------------------------------------------------------------
// Next-token targets and weights of a batch, one thread per position (training/losses.py states the rule): position i is
// supervised by token i + 1 when both are valid, carry the same label and the target is not ignored.  Two adjacent valid
// tokens are in one canonical segment exactly when their labels are the same, so no segments are built here.  One launch
// in the place of about 25 tensor operations of 2 us each.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ long load_integer(const void* x, int bytes, long i) {
  if (bytes == 8) return static_cast<const long*>(x)[i];
  if (bytes == 4) return static_cast<const int*>(x)[i];
  return static_cast<const unsigned char*>(x)[i];
}
__global__ void loss_targets_kernel(const void* __restrict__ ids, int id_bytes, const void* __restrict__ mask, int mask_bytes,
                                    const void* __restrict__ labels, int label_bytes, const float* __restrict__ loss,
                                    int* __restrict__ targets, float* __restrict__ weights, int S, long n, int ignore) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  int target = 0;
  float weight = 0.f;
  if (i % S != S - 1) {
    const long id = load_integer(ids, id_bytes, i + 1);
    bool valid = id != ignore;
    if (mask != nullptr) valid = valid && load_integer(mask, mask_bytes, i) == 1 && load_integer(mask, mask_bytes, i + 1) == 1;
    if (labels != nullptr)
      valid = valid && static_cast<int>(load_integer(labels, label_bytes, i)) == static_cast<int>(load_integer(labels, label_bytes, i + 1));
    weight = valid ? 1.f : 0.f;
    if (loss != nullptr) weight *= loss[i + 1];
    if (weight > 0.f) target = static_cast<int>(id);
  }
  targets[i] = target;
  weights[i] = weight;
}

}  // namespace ew
}  // namespace ctb

using namespace ctb;
using namespace ctb::ew;

static inline int grid_for(long work, int threads, int cap_per_sm = 8) {
  long blocks = (work + threads - 1) / threads;
  const long cap = static_cast<long>(sm_count()) * cap_per_sm;
  if (blocks > cap) blocks = cap;
  return static_cast<int>(blocks < 1 ? 1 : blocks);
}

CTB_API int ctb_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* h_out, float* rstd,
                            int rows, int d, float eps, void* stream) {
  if (d % 8 || d > NORM_MAXV * NORM_THREADS * 8) return fail("rmsnorm: hidden size must be a multiple of 8, <= 16384");
  if (residual && !h_out) return fail("rmsnorm: residual given without h_out");
  const int grid = rows < sm_count() * 8 ? rows : sm_count() * 8;
  // (half of CHAINED_BYTES: us, chained and not, 64 x 4096 2.3 and 2.6, 1000 x 1536 3.3 and 3.7; 4096 x 4096 14.5 and 13.1, with
  // a residual 2000 x 4096 12.0 and 11.2)
  const bool chained = (residual ? 8l : 4l) * rows * d <= CHAINED_BYTES / 2;
  const int nv = (d / 8 + NORM_THREADS - 1) / NORM_THREADS;
#define CTB_NORM_FWD(NV)                                                                                         \
  CTB_CUDA_OK(launch_chained(chained, rmsnorm_fwd_kernel<NV>, grid, NORM_THREADS, 0, stream, 0,                  \
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(residual),                         \
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y), static_cast<__nv_bfloat16*>(h_out),  \
      rstd, rows, d, eps))
  if (nv <= 1) CTB_NORM_FWD(1);
  else if (nv <= 2) CTB_NORM_FWD(2);
  else if (nv <= 4) CTB_NORM_FWD(4);
  else CTB_NORM_FWD(8);
#undef CTB_NORM_FWD
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// Number of per-CTA partial rows the backward kernel writes; `dw_partial` must hold
// ctb_rmsnorm_bwd_parts(rows) * d floats.
CTB_API int ctb_rmsnorm_bwd_parts(int rows) {
  const int cap = sm_count() * 2;
  return rows < cap ? rows : cap;
}

static int launch_dw_reduce(bool chained, const float* partial, int parts, int d, void* dw, int dw_f32, int accumulate,
                            cudaStream_t s) {
  // Few partial rows, as column sums have, leave most of 32 warps idle: column sums of 1000 x 2048 4.9 us with 32, 4.5 with 8, of
  // 1000 x 128256 54.2 and 47.3; a backward norm of 296 partial rows see above.
  const int warps = parts > 96 ? 32 : 8;
  CTB_CUDA_OK(launch_chained(chained, warps == 32 ? rmsnorm_dw_reduce_kernel<32> : rmsnorm_dw_reduce_kernel<8>, (d + 31) / 32,
                             warps * 32, 0, s, 0, partial, parts, d, dw, dw_f32, accumulate));
  return 0;
}

CTB_API int ctb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                            void* dx, float* dw_partial, void* dw, int dw_f32, int dw_accumulate, int rows, int d,
                            void* stream) {
  if (d % 8 || d > NORM_MAXV * NORM_THREADS * 8) return fail("rmsnorm: hidden size must be a multiple of 8, <= 16384");
  const int parts = ctb_rmsnorm_bwd_parts(rows);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool chained = 8l * rows * d <= CHAINED_BYTES;
  const int nv = (d / 8 + NORM_THREADS - 1) / NORM_THREADS;
  // Rows of up to 2048: three blocks fit an SM where two are launched for each, and started early they crowd (us, chained and not: 1000 x
  // 1536 7.3 and 7.0, 2000 x 1536 9.5 and 8.8, 4096 x 1536 14.7 and 12.7); wider ones have no room to (1000 x 4096 8.9 and 9.1, 700
  // x 8192 13.3 and 14.1).  Below 2 MB it is the launch that counts (512 x 256 4.6, unchained 5.5).
#define CTB_NORM_BWD(NV)                                                                       \
  CTB_CUDA_OK(launch_chained(chained && (NV > 1 || 8l * rows * d <= 2l << 20), rmsnorm_bwd_kernel<NV>, parts, NORM_THREADS, 0, s, 0, \
      static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),             \
      static_cast<const __nv_bfloat16*>(w), rstd, static_cast<const __nv_bfloat16*>(dres),     \
      static_cast<__nv_bfloat16*>(dx), dw_partial, rows, d))
  if (nv <= 1) CTB_NORM_BWD(1);
  else if (nv <= 2) CTB_NORM_BWD(2);
  else if (nv <= 4) CTB_NORM_BWD(4);
  else CTB_NORM_BWD(8);
#undef CTB_NORM_BWD
  CTB_CUDA_OK(cudaGetLastError());
  if (dw != nullptr) {
    return launch_dw_reduce(chained, dw_partial, parts, d, dw, dw_f32, dw_accumulate, s);
  }
  return 0;
}

// Rows of partial sums that ctb_column_sum writes for a matrix of `rows` rows and `n` columns.
CTB_API int ctb_column_sum_parts(int rows, int n) {
  const int cols = (n + 255) / 256;
  const int want = (sm_count() * 4 + cols - 1) / cols, most = (rows + 31) / 32;
  return want < most ? want : (most < 1 ? 1 : most);
}
// out[c] (+)= sum over rows of x[r][c]; n and ld multiples of 8 elements, x 16-byte aligned; partial holds
// ctb_column_sum_parts(rows, n) * n floats.
CTB_API int ctb_column_sum(const void* x, long ld, int rows, int n, float* partial, void* out, int out_f32, int accumulate,
                           void* stream) {
  if (n % 8 || ld % 8 || reinterpret_cast<uintptr_t>(x) % 16) return fail("column_sum: rows must be whole 16-byte vectors");
  if (n <= 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int parts = ctb_column_sum_parts(rows, n);
  const bool chained = 2l * rows * n <= CHAINED_BYTES;
  CTB_CUDA_OK(launch_chained(chained, column_sum_kernel, dim3((n + 255) / 256, parts), 256, 0, s, 0,
                             static_cast<const __nv_bfloat16*>(x), ld, rows, n, partial));
  return launch_dw_reduce(chained, partial, parts, n, out, out_f32, accumulate, s);
}

CTB_API int ctb_rope_table(const int* pos, const float* inv_freq, float* cosv, float* sinv, int T, int half,
                           void* stream) {
  rope_table_kernel<<<grid_for(static_cast<long>(T) * half, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      pos, inv_freq, cosv, sinv, T, half);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_rope(void* x, const float* cosv, const float* sinv, long row_stride, int T, int heads, int D, int rot,
                     int style, int inverse, void* stream) {
  if (rot % 2 || rot > D) return fail("rope: rotary_dim must be even and <= head_dim");
  // Whole 16-byte vectors per lane: 8 channels of each half (gpt-neox) or 4 pairs (gpt-j), at most 32 lanes a head.
  // A warp with fewer than 8 lanes in use, or fewer than 10000 vectors in all (16384 where a walk over the heads is
  // long for the number of tokens), is no faster than a thread per pair (us, pair and vector: 8192 tokens, 4 lanes of a warp
  // 3.2 and 4.0; 2048 tokens, 8 lanes 2.7 and 2.4; 333 tokens, 4 heads of 128 2.2 and 2.0; 128 tokens, 10 heads of 128 2.3 and
  // 2.5, 40 heads 3.7 and 2.6).
  // (2 MB and not CHAINED_BYTES: us, chained and not, 512 tokens, 6 heads of 64 1.9 and 2.0; 512, 14 heads of 128 2.6 and 2.3; 2000, 14 heads
  // 5.8 and 4.4; 1000, 40 heads 5.6 and 4.1)
  const bool chained = 4l * T * heads * rot <= 2l << 20;
  const int angles = style == 0 ? 4 : 8;
  const int per_head = rot / 2 / angles;
  if (rot % (2 * angles) == 0 && per_head >= 1 && per_head <= 32 && D % 8 == 0 && row_stride % 8 == 0 &&
      heads * per_head >= 8 && static_cast<long>(T) * heads * per_head >= (T < 256 ? 16384 : 10000) &&
      (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cosv) | reinterpret_cast<uintptr_t>(sinv)) % 16 == 0) {
    const int together = 32 / per_head, walk = (heads + together - 1) / together;
    int share = 0;                 // at most the eight warps of a block (333 tokens, 40 heads of 128: 5.9 us alone, 3.1)
    while (share < 3 && (2 << share) <= walk && (static_cast<long>(T) << share) < sm_count() * 8l) ++share;
    auto kern = style == 0 ? (share ? rope_vec_kernel<0, true> : rope_vec_kernel<0, false>)
                           : (share ? rope_vec_kernel<1, true> : rope_vec_kernel<1, false>);
    CTB_CUDA_OK(launch_chained(chained, kern, grid_for((static_cast<long>(T) << share) * 32, 256), 256, 0, stream, 0,
                               static_cast<__nv_bfloat16*>(x), cosv, sinv, row_stride, T, heads, D, rot, inverse ? -1.f : 1.f,
                               share));
    return 0;
  }
  CTB_CUDA_OK(launch_chained(chained, rope_kernel, grid_for(static_cast<long>(T) * heads * (rot / 2), 256), 256, 0, stream, 0,
                             static_cast<__nv_bfloat16*>(x), cosv, sinv, row_stride, T, heads, D, rot, style,
                             inverse ? -1.f : 1.f));
  return 0;
}

// Blocks an SM.  Calls that move more than L2 holds (126 MB) stream through HBM and go best with several times as many blocks as
// fit at once, backward 24 (us: 16384 x 14336 8: 398, 16: 374, 24: 363 (6.5 TB/s); 8192 x 8960 122, 116, 111), forward 16 (8: 234,
// 16: 231 (6.1 TB/s); 8192 x 8960 79 and 77); others lose by it (1000 x 8960 backward 8: 12.6, 24: 13.3).  Before, with the
// quotient and 8 blocks, 388 and 278 us.
constexpr long SWIGLU_STREAMED = 128l << 20;
CTB_API int ctb_swiglu_fwd(const void* gu, void* h, long T, int f, void* stream) {
  if (f % 8) return fail("swiglu: intermediate size must be a multiple of 8");
  if (T <= 0 || f <= 0) return 0;
  const long total = T * (f / 8);
  const int grid = grid_for(total, 256, 6 * T * f > SWIGLU_STREAMED ? 16 : 8);
  auto kern = total >= 10l * 256 * grid ? swiglu_fwd_kernel<2> : swiglu_fwd_kernel<1>;
  CTB_CUDA_OK(launch_chained(6 * T * f <= CHAINED_BYTES, kern, grid, 256, 0, stream, 0, static_cast<const __nv_bfloat16*>(gu),
                             static_cast<__nv_bfloat16*>(h), T, f));
  return 0;
}

CTB_API int ctb_swiglu_bwd(const void* gu, const void* dh, void* dgu, long T, int f, void* stream) {
  if (f % 8) return fail("swiglu: intermediate size must be a multiple of 8");
  if (T <= 0 || f <= 0) return 0;
  CTB_CUDA_OK(launch_chained(10 * T * f <= CHAINED_BYTES, swiglu_bwd_kernel,
                             grid_for(T * (f / 8), 256, 10 * T * f > SWIGLU_STREAMED ? 24 : 8), 256, 0, stream, 0,
                             static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dh),
                             static_cast<__nv_bfloat16*>(dgu), T, f));
  return 0;
}

CTB_API int ctb_embedding_gather(const int* ids, const void* table, void* out, long T, int d, int vocab,
                                 void* stream) {
  if (d % 8) return fail("embedding: hidden size must be a multiple of 8");
  embedding_gather_kernel<<<grid_for(T * (d / 8), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      ids, static_cast<const __nv_bfloat16*>(table), static_cast<__nv_bfloat16*>(out), T, d, vocab);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_attn_delta(const void* o, const void* dout, float* delta, int B, int S, int H, int D, long o_rs,
                           long do_rs, void* stream) {
  const long warps = static_cast<long>(B) * S * H;
  const int threads = 256;
  const long blocks = (warps * 32 + threads - 1) / threads;
  attn_delta_kernel<<<static_cast<unsigned>(blocks), threads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(dout), delta, B, S, H, D, o_rs, do_rs);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// o, dout: [B,S,H,D] bf16 views (row strides in elements); lse, neg_lse2, neg_delta: [B,H,S] fp32.
CTB_API int ctb_attn_bwd_stats(const void* o, const void* dout, const float* lse, float* neg_lse2, float* neg_delta,
                               int B, int S, int H, int D, long o_rs, long do_rs, void* stream) {
  // 16-byte rows of the two head sizes the flash kernels take, and enough of them: a block of the wide kernel takes
  // 128 rows one after the other, 2.3 us at D = 64 and 3.4 at D = 128 however few there are, where a warp per row
  // (below) takes 1.8 and grows with the rows.  They meet at 64 to 80 D rows (us, warp per row and wide: D = 64 4096 rows
  // 2.5 and 2.4, 8192 rows 3.1 and 2.4, 16384 rows 4.8 and 2.5; D = 128 8192 rows 3.2 and 3.7, 12288 rows 4.6
  // and 4.0, 16384 rows 5.4 and 4.0).  The line stays at 192 D, where 8 heads a block met the warp per row, because the two add
  // in different orders: the last bits of a call do not change with it.
  const long tokens = static_cast<long>(B) * S;
  const bool wide = (D == 64 || D == 128) && o_rs % 8 == 0 && do_rs % 8 == 0 && tokens * H >= 192l * D &&
                    (reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) % 16 == 0;
  const bool chained = attn::chained_rows(tokens, H, D);
  const int head_blocks = (H + STAT_HEADS - 1) / STAT_HEADS;
  if (wide && head_blocks <= 65535) {
    const dim3 grid(static_cast<unsigned>((tokens + STAT_TOKENS - 1) / STAT_TOKENS), head_blocks);
    auto kern = D == 128 ? attn_bwd_stats_vec_kernel<128> : attn_bwd_stats_vec_kernel<64>;
    CTB_CUDA_OK(launch_chained(chained, kern, grid, 256, 0, stream, 0, static_cast<const __nv_bfloat16*>(o),
                               static_cast<const __nv_bfloat16*>(dout), lse, neg_lse2, neg_delta, S, H, tokens, o_rs, do_rs));
    return 0;
  }
  const long warps = static_cast<long>(B) * S * H;
  const int threads = 256;
  const long blocks = (warps * 32 + threads - 1) / threads;
  CTB_CUDA_OK(launch_chained(chained, attn_bwd_stats_kernel, static_cast<unsigned>(blocks), threads, 0, stream, 0,
                             static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(dout), lse, neg_lse2,
                             neg_delta, B, S, H, D, o_rs, do_rs));
  return 0;
}

// block_nll / block_w must hold ceil(rows / 32) floats each; ctb_ce_sums adds them up.  coef = weights * grad_scale * *scale (scale
// may be null).  target_step: see ctb_ce_stats; the logit of a row whose target is outside [0, vocab) counts as 0.
CTB_API int ctb_ce_combine(const float* pmax, const float* psum, int slabs, const float* target_logit, const int* targets,
                           int target_step, int vocab, const float* weights, float grad_scale, const float* scale, float* lse,
                           float* coef, float* block_nll, float* block_w, int rows, void* stream) {
  CTB_CUDA_OK(launch_chained(8l * rows * slabs <= CHAINED_BYTES, ce_combine_kernel, (rows + CE_ROWS - 1) / CE_ROWS,
                             CE_ROWS * CE_WARPS, 0, stream, 0, pmax, psum, slabs, target_logit, targets, target_step, vocab,
                             weights, grad_scale, scale, lse, coef, block_nll, block_w, rows));
  return 0;
}

CTB_API int ctb_ce_sums(const float* block_nll, const float* block_w, int blocks, float* nll, float* w, void* stream) {
  CTB_CUDA_OK(launch_chained(true, ce_sums_kernel, 1, 256, 0, stream, 0, block_nll, block_w, blocks, nll, w));
  return 0;
}

// logits: [rows, vocab] bf16 with row stride ld (elements, multiple of 8); lse/target_logit: [rows].
CTB_API int ctb_logits_ce_stats(const void* logits, long ld, int rows, int vocab, const int* targets, float* lse,
                                float* target_logit, void* stream) {
  if (ld % 8) return fail("logits_ce: row stride must be a multiple of 8 elements");
  if (rows <= 0) return 0;
  logits_ce_stats_kernel<<<rows, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(logits), ld, vocab, targets, lse, target_logit);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_logits_ce_backward(void* logits, long ld, int rows, int vocab, const int* targets, const float* lse,
                                   const float* coef, void* stream) {
  if (ld % 8) return fail("logits_ce: row stride must be a multiple of 8 elements");
  if (rows <= 0) return 0;
  logits_ce_backward_kernel<<<rows, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(logits), ld, vocab, targets, lse, coef);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// The gradient of kept logits in their place (see the kernel): rows of ld fp32 elements become rows of 2 ld bf16 elements.
CTB_API int ctb_kept_logits_gradient(float* logits, long ld, int rows, int vocab, const int* targets, int target_step,
                                     const float* lse, const float* coef, void* stream) {
  if (ld % 8 || vocab % 8 || ld < vocab) return fail("kept_logits: rows must be whole vectors of eight");
  if (rows <= 0) return 0;
  kept_logits_gradient_kernel<<<rows, 256, 0, static_cast<cudaStream_t>(stream)>>>(logits, ld, vocab, targets, target_step, lse,
                                                                                   coef);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// partial must hold ctb_sumsq_parts() floats.
CTB_API int ctb_sumsq_parts() { return sm_count() * 4; }
// round_bf16: square the bf16 rounding of each fp32 element (the norm of gradients "cast to
// the parameter dtype" without materialising the cast).
CTB_API int ctb_sumsq(const void* x, long n, int is_f32, int round_bf16, float* partial, void* stream) {
  const int grid = ctb_sumsq_parts();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (is_f32) sumsq_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(x), n, partial, round_bf16);
  else sumsq_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), n, partial, 0);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

CTB_API int ctb_adamw(void* p, const void* g, int g_f32, void* m, void* v, long n, float lr, float b1, float b2,
                      float eps, float decay, float bc1, float bc2, const float* clip, float gscale, int round_bf16,
                      void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n, 256, 16);
  if (g_f32)
    adamw_kernel<float><<<grid, 256, 0, s>>>(static_cast<__nv_bfloat16*>(p), static_cast<const float*>(g),
                                              static_cast<__nv_bfloat16*>(m), static_cast<__nv_bfloat16*>(v), n, lr,
                                              b1, b2, eps, decay, bc1, bc2, clip, gscale, round_bf16);
  else
    adamw_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<__nv_bfloat16*>(p),
                                                      static_cast<const __nv_bfloat16*>(g),
                                                      static_cast<__nv_bfloat16*>(m), static_cast<__nv_bfloat16*>(v), n,
                                                      lr, b1, b2, eps, decay, bc1, bc2, clip, gscale, 0);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// AdamW over a flat arena of n elements (n % 8 == 0, 16-byte aligned bases) split into nreg
// regions: bounds[nreg + 1] (device, ascending, bounds[0] = 0, bounds[nreg] = n) and
// modes[nreg] (device: 1 decay, 0 no decay, -1 frozen).  One launch.
CTB_API int ctb_adamw_regions(void* p, const void* g, int g_f32, void* m, void* v, long n, const long* bounds,
                              const int* modes, int nreg, float lr, float b1, float b2, float eps, float decay,
                              float bc1, float bc2, const float* clip, float gscale, int round_bf16, void* stream) {
  if (n % 8) return fail("adamw_regions: the arena must be a whole number of 16-byte vectors");
  if (nreg < 1 || nreg > ADAM_MAX_REGIONS) return fail("adamw_regions: between 1 and 512 regions");
  auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
  if (misaligned(p) || misaligned(g) || misaligned(m) || misaligned(v))
    return fail("adamw_regions: parameter, gradient and moment arenas must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n / 8, 256, 8);
  if (g_f32)
    adamw_regions_kernel<float><<<grid, 256, 0, s>>>(
        static_cast<__nv_bfloat16*>(p), static_cast<const float*>(g), static_cast<__nv_bfloat16*>(m),
        static_cast<__nv_bfloat16*>(v), n, bounds, modes, nreg, lr, b1, b2, eps, decay, bc1, bc2, clip, gscale,
        round_bf16);
  else
    adamw_regions_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(
        static_cast<__nv_bfloat16*>(p), static_cast<const __nv_bfloat16*>(g), static_cast<__nv_bfloat16*>(m),
        static_cast<__nv_bfloat16*>(v), n, bounds, modes, nreg, lr, b1, b2, eps, decay, bc1, bc2, clip, gscale, 0);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// idx[k] = k-th row with w != 0 (k < total[0]); block_counts is scratch of ceil(rows / 1024) ints.
CTB_API int ctb_active_rows(const float* w, int rows, int* block_counts, int* idx, int* total, void* stream) {
  if (rows <= 0) return fail("active_rows: no rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int blocks = (rows + ACTIVE_BLOCK - 1) / ACTIVE_BLOCK;
  active_count_kernel<<<blocks, ACTIVE_BLOCK, 0, s>>>(w, rows, block_counts);
  CTB_CUDA_OK(cudaGetLastError());
  active_fill_kernel<<<blocks, ACTIVE_BLOCK, 0, s>>>(w, rows, block_counts, idx, total);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// dst[j, :] = src[idx[j], :] for j < n (bf16 rows of d elements, d % 8 == 0; src has `rows` rows).
CTB_API int ctb_gather_rows(const void* src, long src_stride, int rows, const int* idx, void* dst, long n, int d,
                            void* stream) {
  if (d % 8 || src_stride % 8) return fail("gather_rows: rows must be whole 16-byte vectors");
  if (n <= 0) return 0;
  gather_rows_kernel<<<grid_for(n * (d / 8), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(src), src_stride, idx, static_cast<__nv_bfloat16*>(dst), n, d, rows,
      device_status());
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// dst[idx[j], :] = src[j, :] for j < min(n, total[0]); dst has `rows` rows, those no j names are left alone.
CTB_API int ctb_scatter_rows(const void* src, const int* idx, const int* total, void* dst, long dst_stride, int rows,
                             long n, int d, void* stream) {
  if (d % 8 || dst_stride % 8) return fail("scatter_rows: rows must be whole 16-byte vectors");
  if (n <= 0) return 0;
  scatter_rows_kernel<<<grid_for(n * (d / 8), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(src), idx, total, static_cast<__nv_bfloat16*>(dst), dst_stride, n, d, rows,
      device_status());
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}

// targets / weights [B, S] of the shifted rule.  Integers of 1 (mask only), 4 or 8 bytes; mask, labels and loss may be null.
CTB_API int ctb_loss_targets(const void* ids, int id_bytes, const void* mask, int mask_bytes, const void* labels,
                             int label_bytes, const float* loss, int* targets, float* weights, int B, int S, int ignore,
                             void* stream) {
  const long n = static_cast<long>(B) * S;
  if (n <= 0) return 0;
  loss_targets_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      ids, id_bytes, mask, mask_bytes, labels, label_bytes, loss, targets, weights, S, n, ignore);
  CTB_CUDA_OK(cudaGetLastError());
  return 0;
}
