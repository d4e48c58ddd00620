// Shared pieces of the forward and backward flash-attention kernels.
#pragma once
#include <cudaTypedefs.h>

#include "common.cuh"
#include "runtime.h"

extern "C" int mmt_make_tmap_2d(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                                uint32_t box_inner, uint32_t box_outer);

namespace attn {

constexpr int BQ = 128;   // query rows per tile
constexpr int BKV = 128;  // kv rows per tile
constexpr int kThreads = 192;
constexpr uint32_t CHUNK = 128 * 64 * 2;  // one [128 x 64] bf16 swizzled box = 16 KB
constexpr float LOG2E = 1.4426950408889634f;

struct AttnParams {
  const __nv_bfloat16* qkv;
  __nv_bfloat16* out;          // [T, n_q*dim]
  float* lse;                  // [n_q, T]
  const int* seq_lo;
  const int* seq_hi;
  int T, n_q, n_kv, dim;
  long ld;
  int causal;
  float scale;
  MmtErrorWord* ew;
  // backward only
  const __nv_bfloat16* dout;   // [T, n_q*dim]
  const float* delta;          // [n_q, T]  rowsum(out * dout)
  __nv_bfloat16* dqkv;         // [T, ld]
  float* ws_dk;                // optional [n_q, T, dim] fp32 per-q-head partial dK (GQA: one CTA per q head)
  float* ws_dv;
};

// byte offset of element (row, col) inside a [128 x 64] SW128 box with 128-byte rows
MMT_DEVICE uint32_t sw128_offset(int row, int col) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((((col >> 3) ^ (row & 7)) & 7) << 4) + (col & 7) * 2);
}

// descriptor address of K-step k (16 columns) of a K-major operand whose columns sit in two
// 64-column boxes at `base` and `base + CHUNK`
MMT_DEVICE uint32_t kmajor_kstep_addr(uint32_t base, int k) {
  return base + (k >> 2) * CHUNK + (k & 3) * 32;
}

// K-major operand tile (rows x up-to-128 columns in two boxes): descriptor of K-step k
MMT_DEVICE uint64_t desc_kmajor(uint32_t base, int k) { return make_smem_desc(kmajor_kstep_addr(base, k), 16, 1024); }
// MN-major operand tile: rows are the K dimension (16 rows per step), columns the M/N dimension
MMT_DEVICE uint64_t desc_mnmajor(uint32_t base, int k) { return make_smem_desc(base + k * 2048, CHUNK, 1024); }

// The warps that share a lane quadrant (barriers 1 .. 4): all have read their columns of a score stage before any writes
// P / dS over them.  Nothing else ties the softmax warps together inside a block, so the four quadrants drift apart and
// one quadrant's exponentials run beside another's tensor-memory traffic.
template <int kWarps>
MMT_DEVICE void quadrant_bar_sync(int quadrant) {
  asm volatile("bar.sync %0, %1;" ::"r"(quadrant + 1), "n"(kWarps * 32) : "memory");
}

// Bits i of [lo, hi) within a chunk of 32 columns (lo and hi relative to the chunk's first column).
MMT_DEVICE uint32_t visible_bits(int lo, int hi) {
  const uint32_t below_hi = hi >= 32 ? 0xffffffffu : (hi <= 0 ? 0u : (1u << hi) - 1u);
  const uint32_t below_lo = lo >= 32 ? 0xffffffffu : (lo <= 0 ? 0u : (1u << lo) - 1u);
  return below_hi & ~below_lo;
}

// Largest of three (one instruction; like fmaxf it ignores NaN operands).
MMT_DEVICE float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Two fp32 operations in one instruction (same rounding as the scalar ones).
MMT_DEVICE float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t"
      ".reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "mov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\t"
      "mov.b64 {%0, %1}, d;\n\t"
      "}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
MMT_DEVICE float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t"
      ".reg .b64 a, b, d;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "add.rn.f32x2 d, a, b;\n\t"
      "mov.b64 {%0, %1}, d;\n\t"
      "}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

MMT_DEVICE float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t"
      ".reg .b64 a, b, d;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\t"
      "mov.b64 {%0, %1}, d;\n\t"
      "}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

}  // namespace attn
