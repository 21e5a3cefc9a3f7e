// One decoder layer of a small batch, forward and backward, as one library call each: the launches of
// training/engine.py in the same order with the same arguments, issued from C++.
//
// What it is for: a layer is 9 launches forward and 22 backward of 2 to 10 us of device time each when the batch is small
// (512 tokens of a 256-wide model: 0.25 ms a layer), and from Python each takes 10 to 15 us of host time: a pass
// over two such layers and a 32000-word head took 1.90 ms launch by launch and takes 0.73 ms (host time both).  Large
// batches keep the Python schedule, which gives every intermediate back as soon as it is dead; here they lie in one block
// per call.
//
// Reference counterpart: the scanned decoder block (src/causal_trainer/modeling/architecture.py:275-424).
#include "host_common.h"

CTB_API int ctb_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, float*, int, int, float, void*);
CTB_API int ctb_rmsnorm_bwd_parts(int);
CTB_API int ctb_rmsnorm_bwd(const void*, const void*, const void*, const float*, const void*, void*, float*, void*, int, int,
                            int, int, void*);
CTB_API int ctb_column_sum_parts(int, int);
CTB_API int ctb_column_sum(const void*, long, int, int, float*, void*, int, int, void*);
CTB_API int ctb_rope(void*, const float*, const float*, long, int, int, int, int, int, int, void*);
CTB_API int ctb_swiglu_fwd(const void*, void*, long, int, void*);
CTB_API int ctb_swiglu_bwd(const void*, const void*, void*, long, int, void*);
CTB_API long ctb_gemm_workspace(int, int, int, int, int, int);
CTB_API int ctb_gemm(const void*, const void*, void*, int, int, int, long, long, long, int, int, int, int, float, const void*,
                     int, void*, long, void*);
CTB_API int ctb_attn_fwd_range(const void*, const void*, const void*, void*, float*, const int*, const int*, const int*,
                               const int*, const int*, int, int, int, int, int, int, int, long, long, long, long, float,
                               long long, void*);
CTB_API int ctb_attn_bwd_range(const void*, const void*, const void*, const void*, const void*, const float*, void*, void*,
                               void*, float*, float*, const int*, const int*, const int*, const int*, const int*, const int*,
                               const int*, const int*, const int*, int, int, int, int, int, int, int, long, long, long, long,
                               long, long, long, long, float, long long, void*, long, void*);
CTB_API long ctb_attn_bwd_workspace(int, int, int, int, int, int);

namespace ctb {
namespace layer {

// Mirrored by ops/layer.py (same order, same types).
struct Shape {
  int batch, seq, hidden, q_heads, kv_heads, head_dim, inner, rotary_dim, rope_style, grad_f32;
  int whole_tiles;      // no room in the backward call's block for partial sums of dK / dV (ctb_attn_bwd_workspace)
  float eps, scale;
};
struct Context {
  const float *cosine, *sine;
  const int *seg, *lim, *start, *end, *first_q, *kv_lo, *kv_hi, *q_lo, *q_hi;
};
struct Weights {
  const char *ln1, *ln2, *qkv_w, *qkv_b, *o_w, *gu_w, *down_w;      // (qkv_b may be null)
};

// A block that is cut into pieces; `size` is what the caller holds (0 while the pieces are only counted).
struct Block {
  char* base;
  long size = 0;
  long used = 0;
  bool holds = true;        // the caller's block holds every piece so far
  template <typename T>
  T* take(long count) {
    T* at = reinterpret_cast<T*>(base + used);
    const long end = used + count * static_cast<long>(sizeof(T));
    holds = holds && end <= size;
    used = (end + 255) / 256 * 256;
    return at;
  }
  // The products' workspace: what a counted block asks for, what a real one has left.  A product that finds less than it
  // asked for takes a kernel that needs none, so a switch that is turned between the two costs speed and nothing else.
  char* take_rest(long wanted, long* bytes) {
    *bytes = base == nullptr ? wanted : (size > used ? size - used : 0);
    return take<char>(*bytes);
  }
};

using bf16 = __nv_bfloat16;

struct Sizes {
  long t, qw, kvw, w;
  explicit Sizes(const Shape& s)
      : t(static_cast<long>(s.batch) * s.seq), qw(static_cast<long>(s.q_heads) * s.head_dim),
        kvw(static_cast<long>(s.kv_heads) * s.head_dim), w(qw + 2 * kvw) {}
};

// What a layer keeps for its backward pass, besides its output h.
struct Kept {
  bf16 *x, *qkv, *o, *gu;
  float *rstd1, *rstd2, *lse;
  Kept(const Shape& s, Block& b) {
    const Sizes z(s);
    x = b.take<bf16>(z.t * s.hidden);
    qkv = b.take<bf16>(z.t * z.w);
    o = b.take<bf16>(z.t * z.qw);
    gu = b.take<bf16>(z.t * 2 * s.inner);
    rstd1 = b.take<float>(z.t);
    rstd2 = b.take<float>(z.t);
    lse = b.take<float>(z.t * s.q_heads);
  }
};

long most(long a, long b) { return a > b ? a : b; }

struct Forward {
  bf16 *normed, *branch, *act;
  char* work;
  long work_bytes;
  Forward(const Shape& s, Block& b) {
    const Sizes z(s);
    const int t = static_cast<int>(z.t);
    normed = b.take<bf16>(z.t * s.hidden);
    branch = b.take<bf16>(z.t * s.hidden);
    act = b.take<bf16>(z.t * s.inner);
    long wanted = 0;
    if (b.base == nullptr)
      wanted = most(most(ctb_gemm_workspace(t, static_cast<int>(z.w), s.hidden, 0, 0, 0),
                         ctb_gemm_workspace(t, s.hidden, static_cast<int>(z.qw), 0, 0, 0)),
                    most(ctb_gemm_workspace(t, 2 * s.inner, s.hidden, 0, 0, 0),
                         ctb_gemm_workspace(t, s.hidden, s.inner, 0, 0, 0)));
    work = b.take_rest(wanted, &work_bytes);
  }
};

struct Backward {
  bf16 *act, *n1, *n2, *dact, *dgu, *dn, *dh, *dout_o, *dqkv;
  float *stats, *parts, *no_grad, *rstd;
  char* dkv;
  long dkv_bytes;
  char* work;
  long work_bytes;
  Backward(const Shape& s, Block& b) {
    const Sizes z(s);
    const int t = static_cast<int>(z.t), w = static_cast<int>(z.w), qw = static_cast<int>(z.qw);
    act = b.take<bf16>(z.t * s.inner);
    n1 = b.take<bf16>(z.t * s.hidden);
    n2 = b.take<bf16>(z.t * s.hidden);
    dact = b.take<bf16>(z.t * s.inner);
    dgu = b.take<bf16>(z.t * 2 * s.inner);
    dn = b.take<bf16>(z.t * s.hidden);
    dh = b.take<bf16>(z.t * s.hidden);
    dout_o = b.take<bf16>(z.t * z.qw);
    dqkv = b.take<bf16>(z.t * z.w);
    stats = b.take<float>(2 * z.t * s.q_heads);
    parts = b.take<float>(most(static_cast<long>(ctb_rmsnorm_bwd_parts(t)) * s.hidden,
                               static_cast<long>(ctb_column_sum_parts(t, w)) * w));
    no_grad = b.take<float>(s.hidden);
    rstd = b.take<float>(z.t);
    dkv_bytes = s.whole_tiles ? 0 : ctb_attn_bwd_workspace(s.batch, s.seq, s.seq, s.q_heads, s.kv_heads, s.head_dim);
    dkv = b.take<char>(dkv_bytes);
    long wanted = 0;
    const int shapes[8][3] = {{t, s.inner, s.hidden}, {s.hidden, s.inner, t}, {t, s.hidden, 2 * s.inner},
                              {2 * s.inner, s.hidden, t}, {t, qw, s.hidden}, {s.hidden, qw, t},
                              {t, s.hidden, w}, {w, s.hidden, t}};
    for (int i = 0; i < 8 && b.base == nullptr; ++i)
      wanted = most(wanted, ctb_gemm_workspace(shapes[i][0], shapes[i][1], shapes[i][2], i % 2, i % 2 ? s.grad_f32 : 0, 0));
    work = b.take_rest(wanted, &work_bytes);
  }
};

#define CTB_TRY(expr)              \
  do {                             \
    const int _rc = (expr);        \
    if (_rc != 0) return _rc;      \
  } while (0)

// y[T,out] = x[T,in] W^T (+ bias)
int project(const void* x, const void* w, const void* bias, void* y, long t, long in, long out, char* work, long bytes,
            void* stream) {
  return ctb_gemm(x, w, y, static_cast<int>(t), static_cast<int>(out), static_cast<int>(in), in, in, out, 0, 0, 0, 0, 1.f, bias,
                  0, work, bytes, stream);
}
// dx[T,in] = dy[T,out] W;  dW[out,in] (+)= dy^T x
int project_backward(const void* dy, const void* x, const void* w, void* dx, void* dw, long t, long in, long out, int grad_f32,
                     int accumulate, char* work, long bytes, void* stream) {
  CTB_TRY(ctb_gemm(dy, w, dx, static_cast<int>(t), static_cast<int>(in), static_cast<int>(out), out, in, in, 0, 1, 0, 0, 1.f,
                   nullptr, 0, work, bytes, stream));
  if (dw == nullptr) return 0;
  return ctb_gemm(dy, x, dw, static_cast<int>(out), static_cast<int>(in), static_cast<int>(t), out, in, in, 1, 1, grad_f32,
                  accumulate, 1.f, nullptr, 0, work, bytes, stream);
}

}  // namespace layer
}  // namespace ctb

// Bytes of the kept block, of the forward call's and of the backward call's scratch block, with the GEMM switches as they are.
CTB_API void ctb_layer_bytes(const ctb::layer::Shape* s, long* kept, long* forward, long* backward) {
  using namespace ctb::layer;
  Block k{nullptr}, f{nullptr}, b{nullptr};
  Kept kk(*s, k);
  Forward ff(*s, f);
  Backward bb(*s, b);
  *kept = k.used;
  *forward = f.used;
  *backward = b.used;
}

// h = x + attention branch and mlp, with x = resid + branch (branch null: x = resid, and nothing is kept in x's place).
CTB_API int ctb_layer_forward(const ctb::layer::Shape* sp, const ctb::layer::Context* cx, const ctb::layer::Weights* w,
                              const void* resid, const void* branch, void* kept, long kept_bytes, void* scratch,
                              long scratch_bytes, void* h, void* mlp, void* stream) {
  using namespace ctb::layer;
  const Shape& s = *sp;
  const Sizes z(s);
  const int t = static_cast<int>(z.t);
  if (kept == nullptr || scratch == nullptr) return ctb::fail("layer: no blocks");
  Block kb{static_cast<char*>(kept), kept_bytes}, sb{static_cast<char*>(scratch), scratch_bytes};
  const Kept k(s, kb);
  const Forward f(s, sb);
  if (!kb.holds || !sb.holds) return ctb::fail("layer: a block is too small (ctb_layer_bytes)");
  const void* x = branch != nullptr ? k.x : resid;
  CTB_TRY(ctb_rmsnorm_fwd(resid, branch, w->ln1, f.normed, branch != nullptr ? k.x : nullptr, k.rstd1, t, s.hidden, s.eps, stream));
  CTB_TRY(project(f.normed, w->qkv_w, w->qkv_b, k.qkv, z.t, s.hidden, z.w, f.work, f.work_bytes, stream));
  CTB_TRY(ctb_rope(k.qkv, cx->cosine, cx->sine, z.w, t, s.q_heads + s.kv_heads, s.head_dim, s.rotary_dim, s.rope_style, 0, stream));
  CTB_TRY(ctb_attn_fwd_range(k.qkv, k.qkv + z.qw, k.qkv + z.qw + z.kvw, k.o, k.lse, cx->seg, cx->lim, cx->start, cx->kv_lo,
                             cx->kv_hi, s.batch, s.seq, s.seq, 0, s.q_heads, s.kv_heads, s.head_dim, z.w, z.w, z.w, z.qw, s.scale,
                             0, stream));
  CTB_TRY(project(k.o, w->o_w, nullptr, f.branch, z.t, z.qw, s.hidden, f.work, f.work_bytes, stream));
  CTB_TRY(ctb_rmsnorm_fwd(x, f.branch, w->ln2, f.normed, h, k.rstd2, t, s.hidden, s.eps, stream));
  CTB_TRY(project(f.normed, w->gu_w, nullptr, k.gu, z.t, s.hidden, 2l * s.inner, f.work, f.work_bytes, stream));
  CTB_TRY(ctb_swiglu_fwd(k.gu, f.act, z.t, s.inner, stream));
  return project(f.act, w->down_w, nullptr, mlp, z.t, s.inner, s.hidden, f.work, f.work_bytes, stream);
}

// Gradient dx of the layer's input from the gradient dout of its output h + mlp; the weight gradients go where `g` says (null:
// not wanted).  `x` is the layer's input (resid where there was no branch).
CTB_API int ctb_layer_backward(const ctb::layer::Shape* sp, const ctb::layer::Context* cx, const ctb::layer::Weights* w,
                               const ctb::layer::Weights* grads, int accumulate, const void* x_or_null, const void* h,
                               const void* dout, void* kept, long kept_bytes, void* scratch, long scratch_bytes, void* dx,
                               void* stream) {
  using namespace ctb::layer;
  const Shape& s = *sp;
  const Sizes z(s);
  const int t = static_cast<int>(z.t);
  if (kept == nullptr || scratch == nullptr) return ctb::fail("layer: no blocks");
  Block kb{static_cast<char*>(kept), kept_bytes}, sb{static_cast<char*>(scratch), scratch_bytes};
  const Kept k(s, kb);
  const Backward b(s, sb);
  if (!kb.holds || !sb.holds) return ctb::fail("layer: a block is too small (ctb_layer_bytes)");
  auto at = [](const char* p) { return const_cast<char*>(p); };
  const void* x = x_or_null != nullptr ? x_or_null : k.x;
  // the memory-bound intermediates are cheaper to rebuild than to hold (the inverse norms of the forward pass stay)
  CTB_TRY(ctb_swiglu_fwd(k.gu, b.act, z.t, s.inner, stream));
  CTB_TRY(ctb_rmsnorm_fwd(h, nullptr, w->ln2, b.n2, nullptr, b.rstd, t, s.hidden, s.eps, stream));
  CTB_TRY(ctb_rmsnorm_fwd(x, nullptr, w->ln1, b.n1, nullptr, b.rstd, t, s.hidden, s.eps, stream));
  // MLP branch
  CTB_TRY(project_backward(dout, b.act, w->down_w, b.dact, at(grads->down_w), z.t, s.inner, s.hidden, s.grad_f32, accumulate,
                           b.work, b.work_bytes, stream));
  CTB_TRY(ctb_swiglu_bwd(k.gu, b.dact, b.dgu, z.t, s.inner, stream));
  CTB_TRY(project_backward(b.dgu, b.n2, w->gu_w, b.dn, at(grads->gu_w), z.t, s.hidden, 2l * s.inner, s.grad_f32, accumulate,
                           b.work, b.work_bytes, stream));
  const bool ln2 = grads->ln2 != nullptr, ln1 = grads->ln1 != nullptr;
  CTB_TRY(ctb_rmsnorm_bwd(b.dn, h, w->ln2, k.rstd2, dout, b.dh, b.parts, ln2 ? at(grads->ln2) : reinterpret_cast<char*>(b.no_grad),
                          ln2 ? s.grad_f32 : 1, ln2 ? accumulate : 0, t, s.hidden, stream));
  // attention branch: dh is the gradient of h = x + attn_out
  CTB_TRY(project_backward(b.dh, k.o, w->o_w, b.dout_o, at(grads->o_w), z.t, z.qw, s.hidden, s.grad_f32, accumulate, b.work,
                           b.work_bytes, stream));
  CTB_TRY(ctb_attn_bwd_range(k.qkv, k.qkv + z.qw, k.qkv + z.qw + z.kvw, k.o, b.dout_o, k.lse, b.dqkv, b.dqkv + z.qw,
                             b.dqkv + z.qw + z.kvw, b.stats, b.stats + z.t * s.q_heads, cx->seg, cx->lim, cx->kv_lo, cx->kv_hi,
                             cx->q_lo, cx->q_hi, cx->start, cx->end, cx->first_q, s.batch, s.seq, s.seq, 0, s.q_heads, s.kv_heads,
                             s.head_dim, z.w, z.w, z.w, z.qw, z.qw, z.w, z.w, z.w, s.scale, 0, b.dkv, b.dkv_bytes, stream));
  CTB_TRY(ctb_rope(b.dqkv, cx->cosine, cx->sine, z.w, t, s.q_heads + s.kv_heads, s.head_dim, s.rotary_dim, s.rope_style, 1, stream));
  CTB_TRY(project_backward(b.dqkv, b.n1, w->qkv_w, b.dn, at(grads->qkv_w), z.t, s.hidden, z.w, s.grad_f32, accumulate, b.work,
                           b.work_bytes, stream));
  if (w->qkv_b != nullptr && grads->qkv_b != nullptr)
    CTB_TRY(ctb_column_sum(b.dqkv, z.w, t, static_cast<int>(z.w), b.parts, at(grads->qkv_b), s.grad_f32, accumulate, stream));
  return ctb_rmsnorm_bwd(b.dn, x, w->ln1, k.rstd1, b.dh, dx, b.parts, ln1 ? at(grads->ln1) : reinterpret_cast<char*>(b.no_grad),
                         ln1 ? s.grad_f32 : 1, ln1 ? accumulate : 0, t, s.hidden, stream);
}
