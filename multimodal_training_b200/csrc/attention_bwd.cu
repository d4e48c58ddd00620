// Backward of the packed variable-length flash attention (see attention.cu for the layout).
//
// Three launches, no atomics, deterministic:
//   1. delta[h, t] = sum_d out[t,h,d] * dout[t,h,d]
//   2. dK/dV: one CTA per (128-row KV tile, kv head), looping over the q heads of the GQA group and over blocks
//      of 64 queries that can see the KV tile; transposed scores S^T = K Q^T and dP^T = V dO^T in tensor memory,
//      P^T and dS^T written back over them as packed bf16 and used as tensor-memory A operands of
//      dV += P^T dO and dK += dS^T Q, whose accumulators stay in tensor memory across the whole loop
//   3. dQ: one CTA per (128-row query tile, q head), looping over KV tiles with the same pipeline
//      (dQ += dS K, dS as a tensor-memory operand)
// P = exp(S * scale - lse) and dS = P * (dP - delta) * scale are recomputed from the saved log-sum-exp.
// Every tile is fetched as 64-column TMA boxes that serve as K-major or MN-major operands, so Q, K, V and dO
// need no transposes.  Details at the kernels.
#include "attention_common.cuh"
#include "block_loop.h"

namespace {
using namespace attn;

// ----------------------------------------------------------------------------------------------
// 1. delta
// ----------------------------------------------------------------------------------------------
__global__ void attn_delta_kernel(const __nv_bfloat16* out, const __nv_bfloat16* dout,
                                  float* __restrict__ delta, int T, int n_q, int dim) {
  grid_dependency_sync();
  const long w = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (long)T * n_q) return;
  const long t = w / n_q;
  const int h = (int)(w % n_q);
  const __nv_bfloat16* o = out + t * (long)(n_q * dim) + h * dim;
  const __nv_bfloat16* d = dout + t * (long)(n_q * dim) + h * dim;
  float s = 0.f;
  for (int c = lane * 2; c < dim; c += 64) {
    const float2 a = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(o + c));
    const float2 b = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(d + c));
    s += a.x * b.x + a.y * b.y;
  }
  s = warp_sum(s);
  if (lane == 0) delta[(long)h * T + t] = s;
}

// dK / dV of a GQA group = sum of its q heads' fp32 partials, in head order (deterministic), rounded once.
__global__ void attn_group_reduce_kernel(const float* ws_dk, const float* ws_dv,
                                         __nv_bfloat16* __restrict__ dqkv, int T, int n_q, int n_kv, int dim, long ld) {
  grid_dependency_sync();
  const int group = n_q / n_kv;
  const int per_row = n_kv * dim / 4;                 // float4 items per token and tensor
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)T * per_row * 2) return;
  const int which = (int)(idx / ((long)T * per_row));  // 0 = dK, 1 = dV
  const long rem = idx - (long)which * T * per_row;
  const int t = (int)(rem / per_row);
  const int e = (int)(rem % per_row) * 4;
  const int kvh = e / dim, c = e % dim;
  const float* ws = which ? ws_dv : ws_dk;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int g = 0; g < group; ++g) {
    const float4 v = *reinterpret_cast<const float4*>(ws + ((long)(kvh * group + g) * T + t) * dim + c);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  __nv_bfloat16* dst = dqkv + (long)t * ld + (long)(n_q + which * n_kv + kvh) * dim + c;
  uint2 o;
  o.x = pack_bf16x2(acc.x, acc.y);
  o.y = pack_bf16x2(acc.z, acc.w);
  *reinterpret_cast<uint2*>(dst) = o;
}

// ----------------------------------------------------------------------------------------------
// 2. dK / dV: transposed scores, P^T / dS^T as tensor-memory operands, pipelined.
//
// A kernel that runs its four stages (TMA, S/dP MMAs, softmax, dV/dK MMAs) strictly one after the other and moves
// P and dS through shared memory leaves the tensor core idle most of the time.  Here one CTA owns a 128-row KV
// tile, and
//   * it computes the TRANSPOSED tiles S^T = K Q^T and dP^T = V dO^T for blocks of 64 queries, so the KV rows
//     are the tensor-memory lanes and P^T, dS^T can be written back (packed bf16, tcgen05.st) over the columns
//     they were computed from and fed to dV += P^T dO and dK += dS^T Q as tensor-memory A operands: no P/dS in
//     shared memory, which leaves room for a 3-deep ring of Q/dO blocks;
//   * S^T/dP^T are double buffered in tensor memory (2 x 128 columns) next to dV and dK (128 columns each), so
//     the MMAs of block i+1 run while the softmax warps work on block i;
//   * per-query values (visible range, log-sum-exp, delta) are staged in shared memory by the TMA warp, as far ahead as
//     the Q/dO ring: no softmax warp has a global load or an address in its chain;
//   * S^T and dP^T, and dV and dK, are issued alternately: MMAs that follow one another into ONE accumulator leave
//     bubbles in the tensor pipe, the more so the narrower they are.
//   * sixteen softmax warps (four per scheduler): with eight, the latency of a block's chain was not covered.
// Measured (delta, dK/dV and dQ together, from two barriers and loads in the softmax warps to this): one image of 16384
// patches, 16 heads of 80: 8.28 -> 5.6 ms; one causal sequence of 6144 tokens, 40 / 8 heads of 128: 2.09 -> 1.50 ms.
// What bounds it now: the chain MMA -> tcgen05.ld -> exponentials -> tcgen05.st of a block with two score stages; the
// N = 64 products take about 70 cycles each (they read 6 KB of shared memory).
// Tensor memory: stage s at columns 128 s: S^T [0,64) (P^T over [0,32)), dP^T [64,128) (dS^T over [64,96));
// dV at 256, dK at 384.
// ----------------------------------------------------------------------------------------------
constexpr int BQ2 = 64;                       // queries per block
constexpr uint32_t QBOX = BQ2 * 64 * 2;       // one [64 x 64] bf16 box = 8 KB
constexpr int kRing = 3;
constexpr int kSoftWarps = 16;                // four per lane quadrant, 16 of the 64 score columns each
constexpr int kBwd2Threads = kSoftWarps * 32 + 64;   // and a TMA warp and an MMA warp


template <int DIM>
__global__ void __launch_bounds__(kBwd2Threads, 1)
attn_bwd_dkdv2_kernel(const __grid_constant__ CUtensorMap tm_kv, const __grid_constant__ CUtensorMap tm_q64,
                      const __grid_constant__ CUtensorMap tm_do64, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;                               // 2 boxes of [128 x 64]
  uint8_t* sV = sK + 2 * CHUNK;
  uint8_t* sRing = sV + 2 * CHUNK;                  // kRing x (Q: 2 boxes of [64 x 64], dO: 2 boxes)
  float* sRow = reinterpret_cast<float*>(sRing + kRing * 4 * QBOX);   // [kRing][4][64]: lo, hi, lse*log2e, delta
  int* sFull = reinterpret_cast<int*>(sRow + kRing * 4 * BQ2);    // [kRing]: 1 = no mask
  uint64_t* bars = reinterpret_cast<uint64_t*>(sFull + kRing + 1);
  uint64_t* kv_full = bars;               // 1
  uint64_t* slot_full = bars + 1;         // kRing
  uint64_t* slot_free = bars + 1 + kRing; // kRing
  uint64_t* s_full = bars + 1 + 2 * kRing;   // 2
  uint64_t* pds_full = s_full + 2;           // 2
  uint64_t* row_full = pds_full + 2;         // kRing
  uint64_t* done = row_full + kRing;      // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_kv);
    tma_prefetch_desc(&tm_q64);
    tma_prefetch_desc(&tm_do64);
    mbar_init(kv_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&slot_full[i], 1);
      mbar_init(&slot_free[i], 1);
      mbar_init(&row_full[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&pds_full[i], kSoftWarps);
    }
    mbar_init(done, 1);
    mbar_fence_init();
  }
  if (warp == kSoftWarps + 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  grid_dependency_sync();
  const int kv0 = blockIdx.x * BKV;
  const bool split = p.ws_dk != nullptr;
  const int full_group = p.n_q / p.n_kv;
  const int kv_head = split ? (int)blockIdx.y / full_group : (int)blockIdx.y;
  const int head0 = split ? (int)blockIdx.y : kv_head * full_group;
  const int group = split ? 1 : full_group;
  const int kv_last = min(kv0 + BKV, p.T) - 1;
  const int q_lo = p.causal ? kv0 : p.seq_lo[kv0];
  const int q_hi = p.seq_hi[kv_last];
  const int n_qb = warp_uniform((q_hi - q_lo + BQ2 - 1) / BQ2);
  const int n_iter = n_qb * group;
  const int xk = (p.n_q + kv_head) * DIM, xv = (p.n_q + p.n_kv + kv_head) * DIM;
  const uint32_t t_dv = tmem_base + 256, t_dk = tmem_base + 384;

  if (warp == kSoftWarps) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      mbar_expect_tx(kv_full, 4 * CHUNK);
      tma_load_2d(sK, &tm_kv, kv_full, xk, kv0);
      tma_load_2d(sK + CHUNK, &tm_kv, kv_full, xk + 64, kv0);
      tma_load_2d(sV, &tm_kv, kv_full, xv, kv0);
      tma_load_2d(sV + CHUNK, &tm_kv, kv_full, xv + 64, kv0);
    }
    __syncwarp();
    int head = head0, i = 0;
    const int q_first = warp_uniform(q_lo);
    for (int it = 0; it < n_iter; ++it) {
      const int r0 = q_first + i * BQ2;
      const int r = it % kRing;
      if (!mbar_wait_warp(&slot_free[r], ((it / kRing) & 1) ^ 1, p.ew, 730)) break;
      uint8_t* sQ = sRing + (size_t)r * 4 * QBOX;
      uint8_t* sDO = sQ + 2 * QBOX;
      if (elect_one()) {
        mbar_expect_tx(&slot_full[r], 4 * QBOX);
        tma_load_2d(sQ, &tm_q64, &slot_full[r], head * DIM, r0);
        tma_load_2d(sQ + QBOX, &tm_q64, &slot_full[r], head * DIM + 64, r0);
        tma_load_2d(sDO, &tm_do64, &slot_full[r], head * DIM, r0);
        tma_load_2d(sDO + QBOX, &tm_do64, &slot_full[r], head * DIM + 64, r0);
      }
      __syncwarp();
      // the block's per-query values, two queries per lane.  Their buffer was last read for block it - kRing, whose MMAs
      // (the ones that freed the slot) were issued after every softmax warp had finished it.
      float* rowv = sRow + r * 4 * BQ2;
      bool cover = true;                        // does every query see the whole KV tile?
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = h * 32 + lane, q = r0 + c;
        int lo = 0, hi2 = 0;
        float l2 = 0.f, dl = 0.f;
        if (q < q_hi) {
          lo = p.seq_lo[q];
          hi2 = p.causal ? min(p.seq_hi[q], q + 1) : p.seq_hi[q];
          l2 = p.lse[(long)head * p.T + q] * LOG2E;
          dl = p.delta[(long)head * p.T + q];
        }
        rowv[c] = __int_as_float(lo);
        rowv[BQ2 + c] = __int_as_float(hi2);
        rowv[2 * BQ2 + c] = l2;
        rowv[3 * BQ2 + c] = dl;
        cover = cover && lo <= kv0 && hi2 >= kv0 + BKV;
      }
      cover = __all_sync(0xffffffffu, cover);
      if (lane == 0) {
        sFull[r] = cover ? 1 : 0;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&row_full[r]);
      if (++i == n_qb) { i = 0; ++head; }
    }
  } else if (warp == kSoftWarps + 1) {
    // ------------------------------ MMA issuer ------------------------------
    {
      const uint32_t idesc_1 = make_idesc_bf16(BKV, BQ2, 0, 0);     // S^T, dP^T: M = 128 kv rows, N = 64 queries
      const uint32_t idesc_2 = make_idesc_bf16(BKV, DIM, 0, 1);     // dV, dK: A from tensor memory, B MN-major
      const uint32_t hi = smem_desc_hi(1024);
      const uint32_t k_lo = smem_desc_lo(smem_u32(sK), 16), v_lo = smem_desc_lo(smem_u32(sV), 16);
      const uint32_t ring_k = smem_desc_lo(smem_u32(sRing), 16);       // Q / dO as K-major B of the first MMAs
      const uint32_t ring_mn = smem_desc_lo(smem_u32(sRing), QBOX);    // dO / Q as MN-major B of the second MMAs
      auto mma2 = [&](int j) {
        const uint32_t st = tmem_base + (uint32_t)((j & 1) * 128);
        const uint32_t slot = (uint32_t)(j % kRing) * ((4 * QBOX) >> 4);
        if (!elect_one()) return;
#pragma unroll
        for (int k = 0; k < BQ2 / 16; ++k) {
          // dV += P^T dO, dK += dS^T Q
          tc_mma_ts(t_dv, st + (uint32_t)(k * 8), smem_desc_join(hi, ring_mn + slot + ((2 * QBOX) >> 4) + (uint32_t)(k * 128)),
                    idesc_2, (j | k) != 0);
          tc_mma_ts(t_dk, st + 64u + (uint32_t)(k * 8), smem_desc_join(hi, ring_mn + slot + (uint32_t)(k * 128)), idesc_2,
                    (j | k) != 0);
        }
        tc_commit(&slot_free[j % kRing]);
      };
      bool ok = mbar_wait_warp(kv_full, 0, p.ew, 740);
      for (int it = 0; it < n_iter && ok; ++it) {
        const int r = it % kRing;
        if (!mbar_wait_warp(&slot_full[r], (it / kRing) & 1, p.ew, 741)) { ok = false; break; }
        const uint32_t st = tmem_base + (uint32_t)((it & 1) * 128);
        const uint32_t slot = (uint32_t)r * ((4 * QBOX) >> 4);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < DIM / 16; ++k) {
            const uint32_t a_off = (uint32_t)(((k >> 2) * CHUNK + (k & 3) * 32) >> 4);
            const uint32_t b_off = (uint32_t)(((k >> 2) * QBOX + (k & 3) * 32) >> 4);
            tc_mma_ss(st, smem_desc_join(hi, k_lo + a_off), smem_desc_join(hi, ring_k + slot + b_off), idesc_1, k != 0);
            tc_mma_ss(st + 64u, smem_desc_join(hi, v_lo + a_off), smem_desc_join(hi, ring_k + slot + ((2 * QBOX) >> 4) + b_off),
                      idesc_1, k != 0);
          }
          tc_commit(&s_full[it & 1]);
        }
        __syncwarp();
        if (it > 0) {
          const int j = it - 1;
          if (!mbar_wait_warp(&pds_full[j & 1], (j >> 1) & 1, p.ew, 742)) { ok = false; break; }
          tc_fence_after();
          mma2(j);
          __syncwarp();
        }
      }
      if (ok && n_iter > 0) {
        const int j = n_iter - 1;
        if (mbar_wait_warp(&pds_full[j & 1], (j >> 1) & 1, p.ew, 743)) {
          tc_fence_after();
          mma2(j);
          __syncwarp();
        }
      }
      if (elect_one()) tc_commit(done);
      __syncwarp();
    }
  } else {
    // ------------------------------ softmax warps (16) + epilogue ------------------------------
    const int q4 = warp & 3;               // tensor-memory lane quadrant
    const int part = warp >> 2;            // which 16 of the 64 query columns
    const int row = q4 * 32 + lane;        // kv row of this thread inside the tile
    const int kvrow = kv0 + row;
    const uint32_t lane_addr = ((uint32_t)(q4 * 32) << 16);
    const float sl2 = p.scale * LOG2E;
    const float2 sl2_2 = make_float2(sl2, sl2), scale_2 = make_float2(p.scale, p.scale);
    const auto arrived = [&](int it) {
      return __all_sync(0xffffffffu, mbar_wait(&row_full[it % kRing], (it / kRing) & 1, p.ew, 752) &&
                                         mbar_wait(&s_full[it & 1], (it >> 1) & 1, p.ew, 750)) != 0;
    };
    // all warps of the quadrant have read their columns (P^T / dS^T overwrite them)
    const auto together = [&] { quadrant_bar_sync<kSoftWarps / 4>(q4); };
    const auto work = [&](int it) {
      const int s = it & 1;
      const int buf = it % kRing;
      const float* rowv = sRow + buf * 4 * BQ2;
      tc_fence_after();
      const uint32_t st = tmem_base + lane_addr + (uint32_t)(s * 128);
      uint32_t r_s[16], r_dp[16];
      tmem_ld_32x32b_x16(st + (uint32_t)(part * 16), r_s);
      tmem_ld_32x32b_x16(st + 64u + (uint32_t)(part * 16), r_dp);
      const bool full = sFull[buf] != 0;
      const float4* l2_v = reinterpret_cast<const float4*>(rowv + 2 * BQ2 + part * 16);
      const float4* dl_v = reinterpret_cast<const float4*>(rowv + 3 * BQ2 + part * 16);
      tmem_wait_ld();
      tc_fence_before();
      together();
      tc_fence_after();
      uint32_t pk_p[8], pk_ds[8];
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 l2 = l2_v[i >> 2], dl = dl_v[i >> 2];
        float2 e[2];
        e[0] = fma2(make_float2(__uint_as_float(r_s[i]), __uint_as_float(r_s[i + 1])), sl2_2, make_float2(-l2.x, -l2.y));
        e[1] = fma2(make_float2(__uint_as_float(r_s[i + 2]), __uint_as_float(r_s[i + 3])), sl2_2,
                    make_float2(-l2.z, -l2.w));
        e[0] = make_float2(exp2f(e[0].x), exp2f(e[0].y));
        e[1] = make_float2(exp2f(e[1].x), exp2f(e[1].y));
        if (!full) {
          const int4 lo4 = *reinterpret_cast<const int4*>(rowv + part * 16 + i);
          const int4 hi4 = *reinterpret_cast<const int4*>(rowv + BQ2 + part * 16 + i);
          if (!(kvrow >= lo4.x && kvrow < hi4.x)) e[0].x = 0.f;
          if (!(kvrow >= lo4.y && kvrow < hi4.y)) e[0].y = 0.f;
          if (!(kvrow >= lo4.z && kvrow < hi4.z)) e[1].x = 0.f;
          if (!(kvrow >= lo4.w && kvrow < hi4.w)) e[1].y = 0.f;
        }
        float2 d0 = add2(make_float2(__uint_as_float(r_dp[i]), __uint_as_float(r_dp[i + 1])), make_float2(-dl.x, -dl.y));
        float2 d1 = add2(make_float2(__uint_as_float(r_dp[i + 2]), __uint_as_float(r_dp[i + 3])),
                         make_float2(-dl.z, -dl.w));
        d0 = mul2(mul2(e[0], d0), scale_2);
        d1 = mul2(mul2(e[1], d1), scale_2);
        pk_p[i >> 1] = pack_bf16x2(e[0].x, e[0].y);
        pk_p[(i >> 1) + 1] = pack_bf16x2(e[1].x, e[1].y);
        pk_ds[i >> 1] = pack_bf16x2(d0.x, d0.y);
        pk_ds[(i >> 1) + 1] = pack_bf16x2(d1.x, d1.y);
      }
      tmem_st_32x32b_x8(st + (uint32_t)(part * 8), pk_p);
      tmem_st_32x32b_x8(st + 64u + (uint32_t)(part * 8), pk_ds);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_full[s]);
    };
    bool ok = for_blocks_in_step(n_iter, arrived, work, together);
    // epilogue: thread = kv row; of a quadrant's four warps two write dK and two dV, alternate chunks of 16 columns
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(done, 0, p.ew, 751));
    tc_fence_after();
    const bool is_dk = (part & 1) == 0;
    const uint32_t acc = (is_dk ? t_dk : t_dv) + lane_addr;
    const int xo = is_dk ? xk : xv;
#pragma unroll 1
    for (int c = part >> 1; c < DIM / 16; c += kSoftWarps / 8) {
      uint32_t r[16];
      if (n_iter > 0 && ok) {
        tmem_ld_32x32b_x16(acc + c * 16, r);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0u;
      }
      if (kvrow < p.T && split) {
        float* w = (is_dk ? p.ws_dk : p.ws_dv) + ((long)head0 * p.T + kvrow) * DIM + c * 16;
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(w + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
      } else if (kvrow < p.T) {
        __nv_bfloat16* dst = p.dqkv + (long)kvrow * p.ld + xo + c * 16;
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          uint4 a;
          a.x = pack_bf16x2(__uint_as_float(r[h2 * 8 + 0]), __uint_as_float(r[h2 * 8 + 1]));
          a.y = pack_bf16x2(__uint_as_float(r[h2 * 8 + 2]), __uint_as_float(r[h2 * 8 + 3]));
          a.z = pack_bf16x2(__uint_as_float(r[h2 * 8 + 4]), __uint_as_float(r[h2 * 8 + 5]));
          a.w = pack_bf16x2(__uint_as_float(r[h2 * 8 + 6]), __uint_as_float(r[h2 * 8 + 7]));
          *reinterpret_cast<uint4*>(dst + h2 * 8) = a;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kSoftWarps + 1) tmem_dealloc(tmem_base, 512);
}

constexpr size_t kBwd2Smem = 1024 + 4 * CHUNK + kRing * 4 * QBOX + kRing * 4 * BQ2 * 4 + (kRing + 1) * 4 +
                             (2 + 3 * kRing + 5) * 8 + 16;

// ----------------------------------------------------------------------------------------------
// 3. dQ: same pipeline as the dK/dV kernel above with the roles of Q and KV exchanged.
// One CTA owns a 128-row query tile of one head and walks the visible KV range in blocks of 64 rows:
//   S = Q K_blk^T, dP = dO V_blk^T   (query rows are the tensor-memory lanes, 64 + 64 columns, double buffered)
//   dS = exp2(S*scale*log2e - lse*log2e) * (dP - delta) * scale   (softmax warps as above; per-row values in registers)
//   dQ += dS K_blk                   (dS written as packed bf16 over the dP columns: tensor-memory A operand;
//                                     the K block is the MN-major B operand)
// Tensor memory: stage s at columns 128 s: S [0,64), dP [64,128) (dS over [64,96)); dQ at 256.
// ----------------------------------------------------------------------------------------------
template <int DIM>
__global__ void __launch_bounds__(kBwd2Threads, 1)
attn_bwd_dq2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_kv64, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                               // 2 boxes of [128 x 64]
  uint8_t* sDO = sQ + 2 * CHUNK;
  uint8_t* sRing = sDO + 2 * CHUNK;                 // kRing x (K block: 2 boxes of [64 x 64], V block: 2 boxes)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRing + kRing * 4 * QBOX);
  uint64_t* q_full = bars;                // 1
  uint64_t* slot_full = bars + 1;         // kRing
  uint64_t* slot_free = bars + 1 + kRing; // kRing
  uint64_t* s_full = bars + 1 + 2 * kRing;   // 2
  uint64_t* ds_full = s_full + 2;            // 2
  uint64_t* done = ds_full + 2;              // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_kv64);
    mbar_init(q_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&slot_full[i], 1);
      mbar_init(&slot_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&ds_full[i], kSoftWarps);
    }
    mbar_init(done, 1);
    mbar_fence_init();
  }
  if (warp == kSoftWarps + 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  grid_dependency_sync();
  // causal: the last query tiles see the most KV blocks and are started first
  const int q0 = (p.causal ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x) * BQ;
  const int head = blockIdx.y;
  const int kv_head = head / (p.n_q / p.n_kv);
  const int q_last = min(q0 + BQ, p.T) - 1;
  const int kv_lo = p.seq_lo[q0];
  const int kv_hi = p.causal ? min(p.seq_hi[q_last], q_last + 1) : p.seq_hi[q_last];
  const int n_iter = warp_uniform((kv_hi - kv_lo + BQ2 - 1) / BQ2);
  const int xq = head * DIM, xk = (p.n_q + kv_head) * DIM, xv = (p.n_q + p.n_kv + kv_head) * DIM;
  const uint32_t t_dq = tmem_base + 256;

  if (warp == kSoftWarps) {
    if (elect_one()) {
      mbar_expect_tx(q_full, 4 * CHUNK);
      tma_load_2d(sQ, &tm_q, q_full, xq, q0);
      tma_load_2d(sQ + CHUNK, &tm_q, q_full, xq + 64, q0);
      tma_load_2d(sDO, &tm_do, q_full, xq, q0);
      tma_load_2d(sDO + CHUNK, &tm_do, q_full, xq + 64, q0);
    }
    __syncwarp();
    const int kv_first = warp_uniform(kv_lo);
    for (int it = 0; it < n_iter; ++it) {
      const int r0 = kv_first + it * BQ2;
      const int r = it % kRing;
      if (!mbar_wait_warp(&slot_free[r], ((it / kRing) & 1) ^ 1, p.ew, 760)) break;
      uint8_t* sKb = sRing + (size_t)r * 4 * QBOX;
      uint8_t* sVb = sKb + 2 * QBOX;
      if (elect_one()) {
        mbar_expect_tx(&slot_full[r], 4 * QBOX);
        tma_load_2d(sKb, &tm_kv64, &slot_full[r], xk, r0);
        tma_load_2d(sKb + QBOX, &tm_kv64, &slot_full[r], xk + 64, r0);
        tma_load_2d(sVb, &tm_kv64, &slot_full[r], xv, r0);
        tma_load_2d(sVb + QBOX, &tm_kv64, &slot_full[r], xv + 64, r0);
      }
      __syncwarp();
    }
  } else if (warp == kSoftWarps + 1) {
    {
      const uint32_t idesc_1 = make_idesc_bf16(BQ, BQ2, 0, 0);      // S, dP: M = 128 queries, N = 64 kv rows
      const uint32_t idesc_2 = make_idesc_bf16(BQ, DIM, 0, 1);      // dQ: A from tensor memory, B = K block MN-major
      const uint32_t hi = smem_desc_hi(1024);
      const uint32_t q_lo = smem_desc_lo(smem_u32(sQ), 16), do_lo = smem_desc_lo(smem_u32(sDO), 16);
      const uint32_t ring_k = smem_desc_lo(smem_u32(sRing), 16);
      const uint32_t ring_mn = smem_desc_lo(smem_u32(sRing), QBOX);
      auto mma2 = [&](int j) {
        const uint32_t st = tmem_base + (uint32_t)((j & 1) * 128);
        const uint32_t slot = (uint32_t)(j % kRing) * ((4 * QBOX) >> 4);
        if (!elect_one()) return;
#pragma unroll
        for (int k = 0; k < BQ2 / 16; ++k)
          tc_mma_ts(t_dq, st + 64u + (uint32_t)(k * 8), smem_desc_join(hi, ring_mn + slot + (uint32_t)(k * 128)), idesc_2,
                    (j | k) != 0);
        tc_commit(&slot_free[j % kRing]);
      };
      bool ok = mbar_wait_warp(q_full, 0, p.ew, 770);
      for (int it = 0; it < n_iter && ok; ++it) {
        const int r = it % kRing;
        if (!mbar_wait_warp(&slot_full[r], (it / kRing) & 1, p.ew, 771)) { ok = false; break; }
        const uint32_t st = tmem_base + (uint32_t)((it & 1) * 128);
        const uint32_t slot = (uint32_t)r * ((4 * QBOX) >> 4);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < DIM / 16; ++k) {
            const uint32_t a_off = (uint32_t)(((k >> 2) * CHUNK + (k & 3) * 32) >> 4);
            const uint32_t b_off = (uint32_t)(((k >> 2) * QBOX + (k & 3) * 32) >> 4);
            tc_mma_ss(st, smem_desc_join(hi, q_lo + a_off), smem_desc_join(hi, ring_k + slot + b_off), idesc_1, k != 0);
            tc_mma_ss(st + 64u, smem_desc_join(hi, do_lo + a_off), smem_desc_join(hi, ring_k + slot + ((2 * QBOX) >> 4) + b_off),
                      idesc_1, k != 0);
          }
          tc_commit(&s_full[it & 1]);
        }
        __syncwarp();
        if (it > 0) {
          const int j = it - 1;
          if (!mbar_wait_warp(&ds_full[j & 1], (j >> 1) & 1, p.ew, 772)) { ok = false; break; }
          tc_fence_after();
          mma2(j);
          __syncwarp();
        }
      }
      if (ok && n_iter > 0) {
        const int j = n_iter - 1;
        if (mbar_wait_warp(&ds_full[j & 1], (j >> 1) & 1, p.ew, 773)) {
          tc_fence_after();
          mma2(j);
          __syncwarp();
        }
      }
      if (elect_one()) tc_commit(done);
      __syncwarp();
    }
  } else {
    const int q4 = warp & 3;
    const int part = warp >> 2;            // which 16 of the 64 kv columns
    const int row = q4 * 32 + lane;
    const int qrow = q0 + row;
    const bool row_ok = qrow < p.T;
    const uint32_t lane_addr = ((uint32_t)(q4 * 32) << 16);
    const float sl2 = p.scale * LOG2E;
    int lo = 0, hi2 = 0;
    float lse_l2 = 0.f, delta = 0.f;
    if (row_ok) {
      lo = p.seq_lo[qrow];
      hi2 = p.seq_hi[qrow];
      if (p.causal) hi2 = min(hi2, qrow + 1);
      lse_l2 = p.lse[(long)head * p.T + qrow] * LOG2E;
      delta = p.delta[(long)head * p.T + qrow];
    }
    const float2 sl2_2 = make_float2(sl2, sl2), scale_2 = make_float2(p.scale, p.scale);
    const float2 lse_2 = make_float2(-lse_l2, -lse_l2), delta_2 = make_float2(-delta, -delta);
    const auto arrived = [&](int it) {
      return __all_sync(0xffffffffu, mbar_wait(&s_full[it & 1], (it >> 1) & 1, p.ew, 780)) != 0;
    };
    // all warps of the quadrant have read their dP columns before dS overwrites them
    const auto together = [&] { quadrant_bar_sync<kSoftWarps / 4>(q4); };
    const auto work = [&](int it) {
      const int s = it & 1;
      const int kvb = kv_lo + it * BQ2 + part * 16;          // first kv row of this warp's 16 columns
      tc_fence_after();
      const uint32_t st = tmem_base + lane_addr + (uint32_t)(s * 128);
      uint32_t r_s[16], r_dp[16];
      tmem_ld_32x32b_x16(st + (uint32_t)(part * 16), r_s);
      tmem_ld_32x32b_x16(st + 64u + (uint32_t)(part * 16), r_dp);
      const bool full = __all_sync(0xffffffffu, kvb >= lo && kvb + 16 <= hi2);
      tmem_wait_ld();
      tc_fence_before();
      together();
      tc_fence_after();
      uint32_t pk_ds[8];
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        float2 e = fma2(make_float2(__uint_as_float(r_s[i]), __uint_as_float(r_s[i + 1])), sl2_2, lse_2);
        e = make_float2(exp2f(e.x), exp2f(e.y));
        if (!full) {
          const int kv = kvb + i;
          if (!(kv >= lo && kv < hi2)) e.x = 0.f;
          if (!(kv + 1 >= lo && kv + 1 < hi2)) e.y = 0.f;
        }
        float2 d = add2(make_float2(__uint_as_float(r_dp[i]), __uint_as_float(r_dp[i + 1])), delta_2);
        d = mul2(mul2(e, d), scale_2);
        pk_ds[i >> 1] = pack_bf16x2(d.x, d.y);
      }
      tmem_st_32x32b_x8(st + 64u + (uint32_t)(part * 8), pk_ds);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_full[s]);
    };
    bool ok = for_blocks_in_step(n_iter, arrived, work, together);
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(done, 0, p.ew, 781));
    tc_fence_after();
    // epilogue: the warps of a lane quadrant split the head's columns in 16-column chunks
    __nv_bfloat16* dst = p.dqkv + (long)qrow * p.ld + xq;
#pragma unroll 1
    for (int c = part; c < DIM / 16; c += kSoftWarps / 4) {
      uint32_t r[16];
      if (n_iter > 0 && ok) {
        tmem_ld_32x32b_x16(t_dq + lane_addr + c * 16, r);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0u;
      }
      if (row_ok) {
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          uint4 a;
          a.x = pack_bf16x2(__uint_as_float(r[h2 * 8 + 0]), __uint_as_float(r[h2 * 8 + 1]));
          a.y = pack_bf16x2(__uint_as_float(r[h2 * 8 + 2]), __uint_as_float(r[h2 * 8 + 3]));
          a.z = pack_bf16x2(__uint_as_float(r[h2 * 8 + 4]), __uint_as_float(r[h2 * 8 + 5]));
          a.w = pack_bf16x2(__uint_as_float(r[h2 * 8 + 6]), __uint_as_float(r[h2 * 8 + 7]));
          *reinterpret_cast<uint4*>(dst + c * 16 + h2 * 8) = a;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kSoftWarps + 1) tmem_dealloc(tmem_base, 512);
}

constexpr size_t kDq2Smem = 1024 + 4 * CHUNK + kRing * 4 * QBOX + (2 + 2 * kRing + 5) * 8 + 16;

template <int DIM>
int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tq64, const CUtensorMap& tdo64,
               const AttnParams& p, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_dkdv2_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kBwd2Smem);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(attn_bwd_dq2_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDq2Smem);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  const int tiles = (p.T + BQ - 1) / BQ;
  launch_dependent(attn_bwd_dkdv2_kernel<DIM>, dim3(tiles, p.ws_dk ? p.n_q : p.n_kv), kBwd2Threads, kBwd2Smem, st,
                     tq, tq64, tdo64, p);
  if (p.ws_dk) {
    const long items = (long)p.T * (p.n_kv * DIM / 4) * 2;
    launch_dependent(attn_group_reduce_kernel, (unsigned)((items + 255) / 256), 256, 0, st,
                     p.ws_dk, p.ws_dv, p.dqkv, p.T, p.n_q,
                                                                             p.n_kv, DIM, p.ld);
  }
  launch_dependent(attn_bwd_dq2_kernel<DIM>, dim3(tiles, p.n_q), kBwd2Threads, kDq2Smem, st,
                     tq, tdo, tq64, p);
  return (int)cudaGetLastError();
}

}  // namespace

// dqkv [T, ld] receives dq | dk | dv in the layout of qkv.  delta is fp32 scratch [n_q, T].  ws is optional fp32
// scratch of 2 * n_q * T * dim floats: with it (and n_q > n_kv) dK/dV run one CTA per q head and are summed over
// each GQA group afterwards, which fills the GPU when there are few KV tiles.
extern "C" int mmt_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                            void* dqkv, const int* seq_lo, const int* seq_hi, long T, int n_q, int n_kv, int dim,
                            long ld, int causal, float scale, float* ws, void* stream) {
  if (T <= 0) return 0;
  if (mmt_ensure_context(qkv)) return -7;
  if ((dim != 80 && dim != 128) || n_q % n_kv || (ld & 7)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  {
    const long warps = T * n_q;
    const int threads = 256;
    const long blocks = (warps * 32 + threads - 1) / threads;
    launch_dependent(attn_delta_kernel, (unsigned)blocks, threads, 0, st,
                     reinterpret_cast<const __nv_bfloat16*>(out),
                                                           reinterpret_cast<const __nv_bfloat16*>(dout), delta,
                                                           (int)T, n_q, dim);
  }
  CUtensorMap tq, tdo;
  const uint64_t width = (uint64_t)(n_q + 2 * n_kv) * dim;
  int r = mmt_make_tmap_2d(&tq, qkv, width, (uint64_t)T, (uint64_t)ld, 64, 128);
  if (r) return 1000 + r;
  r = mmt_make_tmap_2d(&tdo, dout, (uint64_t)n_q * dim, (uint64_t)T, (uint64_t)n_q * dim, 64, 128);
  if (r) return 2000 + r;
  AttnParams p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  p.out = nullptr;
  p.lse = const_cast<float*>(lse);
  p.seq_lo = seq_lo;
  p.seq_hi = seq_hi;
  p.T = (int)T; p.n_q = n_q; p.n_kv = n_kv; p.dim = dim; p.ld = ld;
  p.causal = causal; p.scale = scale;
  p.ew = mmt_error_word();
  p.dout = reinterpret_cast<const __nv_bfloat16*>(dout);
  p.delta = delta;
  p.dqkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  const bool split = ws != nullptr && n_q > n_kv;
  p.ws_dk = split ? ws : nullptr;
  p.ws_dv = split ? ws + (long)n_q * T * dim : nullptr;
  CUtensorMap tq64, tdo64;   // 64-row boxes: the query blocks of dK/dV, the KV blocks of dQ
  r = mmt_make_tmap_2d(&tq64, qkv, width, (uint64_t)T, (uint64_t)ld, 64, 64);
  if (r) return 3000 + r;
  r = mmt_make_tmap_2d(&tdo64, dout, (uint64_t)n_q * dim, (uint64_t)T, (uint64_t)n_q * dim, 64, 64);
  if (r) return 4000 + r;
  return dim == 80 ? launch_bwd<80>(tq, tdo, tq64, tdo64, p, st) : launch_bwd<128>(tq, tdo, tq64, tdo64, p, st);
}
