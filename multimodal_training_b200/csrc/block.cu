// One transformer block per call: the host side of ops/blocks.py in native code.
//
// A block is 9 launches forward and up to 21 backward.  Issued one by one from Python (a ctypes call with up to 21
// arguments, an output allocation and several tensor lookups each) a launch costs 15-20 us of host time, which is more
// than many of these kernels run: at 256 patches the vision encoder took 6.3 ms for 3.6 ms of device work.  Here a
// block is one call with one array of addresses.
//
// The order of the kernels, their arguments and their rounding points are those of the per-op graph.
#include <cstdint>

#include "runtime.h"

extern "C" {
int mmt_rmsnorm_fwd(const void*, const void*, void*, float*, long, int, float, void*);
int mmt_rmsnorm_bwd_parts(long);
int mmt_rmsnorm_bwd_add_partial(const void*, const void*, const void*, const float*, const void*, void*, float*, long, int,
                                int*, void*);
int mmt_rope(void*, const float*, const float*, long, int, int, long, int, void*);
int mmt_swiglu_fwd(const void*, void*, long, int, void*);
int mmt_swiglu_bwd(const void*, const void*, void*, long, int, void*);
int mmt_colsum_parts(long);
int mmt_colsum_partial(const void*, float*, long, int, long, void*);
int mmt_reduce_partials(const MmtReduceSegment*, int, void*);
int mmt_gemm_bf16(const void*, const void*, void*, const void*, const void*, int, int, int, int, int, int, int, int, int,
                  int, int, int, float, int, void*);
int mmt_attn_fwd(const void*, void*, float*, const int*, const int*, long, int, int, int, long, int, float, void*);
int mmt_attn_local_fwd(const void*, void*, float*, const int*, const int*, const int*, int, long, int, int, int, long,
                       int, float, void*);
int mmt_attn_local_bwd(const void*, const void*, const void*, const float*, void*, const int*, const int*, const int*, int,
                       long, int, int, int, long, int, float, void*);
int mmt_attn_bwd(const void*, const void*, const void*, const float*, float*, void*, const int*, const int*, long, int,
                 int, int, long, int, float, float*, void*);
}

namespace {

// The argument array; ops/blocks.py builds it in this order.  Weights, then (behind the rest) weight gradients in the
// same order; biases may be 0.
enum Weight { LN1, QKV_W, QKV_B, PROJ_W, PROJ_B, LN2, GU_W, GU_B, DOWN_W, DOWN_B, N_WEIGHTS };
struct BlockArgs {
  uint64_t w[N_WEIGHTS];
  uint64_t x, y;                 // block input and output (backward: y unused)
  uint64_t cos, sin, lo, hi;
  uint64_t h1, rstd1, qkv, a, lse, x1, h2, rstd2, gu, m;   // activations [T, ...]; backward reads them
  int64_t T, C, n_q, n_kv, dim, rope_heads, inter, causal;
  uint64_t packs;                // packs of short sequences, or 0
  int64_t n_packs;
  // backward only
  uint64_t g[N_WEIGHTS];
  int64_t accumulate;            // bit i: add to g[i]
  uint64_t dy, dx;
  uint64_t dgu, big, mid, dx1;   // scratch: [T, 2 inter], [T, max(inter, qkv width)], [T, max(C, n_q dim)], [T, C]
  uint64_t delta, ws, part;      // attention scratch (ws may be 0); fp32 partial sums of norms and biases, one after the other
  int64_t launches;              // out: kernels launched
};
static_assert(sizeof(BlockArgs) % 8 == 0, "an array of 64-bit words");

struct Issue {
  BlockArgs& b;
  void* st;
  int rc = 0;
  // partial sums of biases and norm weights, finished by one launch at the end of backward
  MmtReduceSegment sums[MMT_MAX_REDUCE_SEGMENTS];
  int n_sums = 0;
  long part_used = 0;            // floats of b.part in use
  float* partial_rows(int wi, int parts, long cols) {
    float* at = f(b.part) + part_used;
    part_used += (long)parts * cols;
    sums[n_sums++] = MmtReduceSegment{at, p(b.g[wi]), parts, (int)cols, acc(wi)};
    return at;
  }
  void* p(uint64_t v) const { return reinterpret_cast<void*>(v); }
  float* f(uint64_t v) const { return reinterpret_cast<float*>(v); }
  const int* i(uint64_t v) const { return reinterpret_cast<const int*>(v); }
  int acc(int wi) const { return (int)(b.accumulate >> wi & 1); }
  void done(int code, int launches) {
    if (rc == 0) rc = code;
    b.launches += launches;
  }
  // y[T, n] = x[T, k] w[n, k]^T (+ bias) (+ residual)
  void linear(uint64_t x, uint64_t w, uint64_t bias, uint64_t res, uint64_t y, long n, long k) {
    if (rc) return;
    done(mmt_gemm_bf16(p(x), p(w), p(y), p(bias), p(res), (int)b.T, (int)n, (int)k, (int)k, (int)k, (int)n,
                       res ? (int)n : 0, 0, 0, 0, 0, 0, 1.f, 0, st), 1);
  }
  // gradients of that layer: dw, db into the parameters' buffers, dx[T, k] = dy w
  void linear_bwd(uint64_t dy, uint64_t x, int wi, uint64_t dx, long n, long k) {
    if (rc) return;
    done(mmt_gemm_bf16(p(dy), p(x), p(b.g[wi]), nullptr, nullptr, (int)n, (int)k, (int)b.T, (int)n, (int)k, (int)k, 0, 1,
                       1, 0, acc(wi), 0, 1.f, 0, st), 1);
    if (!rc && b.w[wi + 1])
      done(mmt_colsum_partial(p(dy), partial_rows(wi + 1, mmt_colsum_parts(b.T), n), b.T, (int)n, n, st), 1);
    if (rc) return;
    done(mmt_gemm_bf16(p(dy), p(b.w[wi]), p(dx), nullptr, nullptr, (int)b.T, (int)k, (int)n, (int)n, (int)k, (int)k, 0, 0,
                       1, 0, 0, 0, 1.f, 0, st), 1);
  }
  void norm(uint64_t x, int wi, uint64_t y, uint64_t rstd, float eps) {
    if (rc) return;
    done(mmt_rmsnorm_fwd(p(x), p(b.w[wi]), p(y), f(rstd), b.T, (int)b.C, eps, st), 1);
  }
  void norm_bwd(uint64_t dy, uint64_t x, int wi, uint64_t rstd, uint64_t extra, uint64_t dx) {
    if (rc) return;
    float* at = partial_rows(wi, mmt_rmsnorm_bwd_parts(b.T), b.C);
    done(mmt_rmsnorm_bwd_add_partial(p(dy), p(x), p(b.w[wi]), f(rstd), p(extra), p(dx), at, b.T, (int)b.C,
                                     &sums[n_sums - 1].parts, st), 1);
  }
  void rope(uint64_t t, int inverse) {
    if (rc) return;
    done(mmt_rope(p(t), f(b.cos), f(b.sin), b.T, (int)b.rope_heads, (int)b.dim, (b.n_q + 2 * b.n_kv) * b.dim, inverse,
                  st), 1);
  }
  void swiglu() {
    if (rc) return;
    done(mmt_swiglu_fwd(p(b.gu), p(b.m), b.T, (int)b.inter, st), 1);
  }
};

}  // namespace

extern "C" {

// Number of 64-bit words of the argument array.
int mmt_block_words() { return (int)(sizeof(BlockArgs) / 8); }

// x1 = x + proj(attention(rope(qkv(norm(x))))), y = x1 + down(swiglu(gate_up(norm(x1)))).
// `y` == 0: everything but the last projection (what a backward that recomputes needs).
int mmt_block_fwd(int64_t* words, float eps, float scale, void* stream) {
  BlockArgs& b = *reinterpret_cast<BlockArgs*>(words);
  b.launches = 0;
  if (b.T <= 0) return 0;
  if (mmt_ensure_context(reinterpret_cast<const void*>(b.x))) return -7;
  Issue s{b, stream};
  const long qw = (b.n_q + 2 * b.n_kv) * b.dim, aw = b.n_q * b.dim;
  s.norm(b.x, LN1, b.h1, b.rstd1, eps);
  s.linear(b.h1, b.w[QKV_W], b.w[QKV_B], 0, b.qkv, qw, b.C);
  s.rope(b.qkv, 0);
  if (!s.rc && b.packs)
    s.done(mmt_attn_local_fwd(s.p(b.qkv), s.p(b.a), s.f(b.lse), s.i(b.lo), s.i(b.hi), s.i(b.packs), (int)b.n_packs, b.T,
                              (int)b.n_q, (int)b.n_kv, (int)b.dim, qw, (int)b.causal, scale, stream), 1);
  else if (!s.rc)
    s.done(mmt_attn_fwd(s.p(b.qkv), s.p(b.a), s.f(b.lse), s.i(b.lo), s.i(b.hi), b.T, (int)b.n_q, (int)b.n_kv, (int)b.dim,
                        qw, (int)b.causal, scale, stream), 1);
  s.linear(b.a, b.w[PROJ_W], b.w[PROJ_B], b.x, b.x1, b.C, aw);
  s.norm(b.x1, LN2, b.h2, b.rstd2, eps);
  s.linear(b.h2, b.w[GU_W], b.w[GU_B], 0, b.gu, 2 * b.inter, b.C);
  s.swiglu();
  if (b.y) s.linear(b.m, b.w[DOWN_W], b.w[DOWN_B], b.x1, b.y, b.C, b.inter);
  return s.rc;
}

// The element-wise intermediates h1, h2 and m from x, x1 and gu.
int mmt_block_rebuild(int64_t* words, float eps, void* stream) {
  BlockArgs& b = *reinterpret_cast<BlockArgs*>(words);
  b.launches = 0;
  if (b.T <= 0) return 0;
  if (mmt_ensure_context(reinterpret_cast<const void*>(b.x))) return -7;
  Issue s{b, stream};
  s.norm(b.x, LN1, b.h1, b.rstd1, eps);
  s.norm(b.x1, LN2, b.h2, b.rstd2, eps);
  s.swiglu();
  return s.rc;
}

// Gradients of all parameters and of x, from dy and the activations.
int mmt_block_bwd(int64_t* words, float scale, void* stream) {
  BlockArgs& b = *reinterpret_cast<BlockArgs*>(words);
  b.launches = 0;
  if (b.T <= 0) return 0;
  if (mmt_ensure_context(reinterpret_cast<const void*>(b.x))) return -7;
  Issue s{b, stream};
  const long qw = (b.n_q + 2 * b.n_kv) * b.dim, aw = b.n_q * b.dim;
  // MLP half
  s.linear_bwd(b.dy, b.m, DOWN_W, b.big, b.C, b.inter);
  if (!s.rc) s.done(mmt_swiglu_bwd(s.p(b.big), s.p(b.gu), s.p(b.dgu), b.T, (int)b.inter, stream), 1);
  s.linear_bwd(b.dgu, b.h2, GU_W, b.mid, 2 * b.inter, b.C);
  s.norm_bwd(b.mid, b.x1, LN2, b.rstd2, b.dy, b.dx1);
  // attention half
  s.linear_bwd(b.dx1, b.a, PROJ_W, b.mid, b.C, aw);
  if (!s.rc && b.packs && b.n_q == b.n_kv)
    s.done(mmt_attn_local_bwd(s.p(b.qkv), s.p(b.a), s.p(b.mid), s.f(b.lse), s.p(b.big), s.i(b.lo), s.i(b.hi),
                              s.i(b.packs), (int)b.n_packs, b.T, (int)b.n_q, (int)b.n_kv, (int)b.dim, qw, (int)b.causal,
                              scale, stream), 1);
  else if (!s.rc)
    s.done(mmt_attn_bwd(s.p(b.qkv), s.p(b.a), s.p(b.mid), s.f(b.lse), s.f(b.delta), s.p(b.big), s.i(b.lo), s.i(b.hi), b.T,
                        (int)b.n_q, (int)b.n_kv, (int)b.dim, qw, (int)b.causal, scale, s.f(b.ws), stream),
           b.ws ? 4 : 3);
  s.rope(b.big, 1);
  s.linear_bwd(b.big, b.h1, QKV_W, b.mid, qw, b.C);
  s.norm_bwd(b.mid, b.x, LN1, b.rstd1, b.dx1, b.dx);
  if (!s.rc) s.done(mmt_reduce_partials(s.sums, s.n_sums, stream), 1);
  return s.rc;
}

}  // extern "C"
