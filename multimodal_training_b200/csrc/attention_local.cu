// Attention over short sequences: packs of whole sequences of up to 128 rows together (the vision encoder's windows).
//
// The kernels of attention.cu and attention_bwd.cu walk KV blocks for a 128-row query tile.  When no sequence reaches out
// of its tile there is nothing to walk: one CTA sees every query and every key of its rows.  So
//   * forward needs one S and one PV product, 97 KB of shared memory and half of tensor memory: two CTAs per SM hide
//     each other's load, softmax and store phases (the general kernel has one CTA per SM);
//   * backward computes P and dS ONCE and takes all three gradients from them (five products where the dK/dV and dQ
//     kernels need seven), reads Q, K, V and dO once, and forms delta = rowsum(out * dout) itself: one launch for three.
// Measured in the kernels' own time, 64-row windows, 16384 patches, 16 heads of 80: forward 72.6 -> 50 us, backward
// 276 -> 141 us; vision step of a 1792 x 1792 image 125.4 -> 121.7 ms.
//
// `items` holds (first row, rows) of every pack.  Packs are whole 128-row tiles (the last one may be shorter): batches in
// which a sequence lies across a multiple of 128 rows go to the general kernels.  So every sum here runs over the same
// keys in the same order as there, and a batch gives the same bits on both paths.  (Packs cut elsewhere were 5 % faster
// for a step on photos, but a row's probabilities were then rounded relative to another maximum, and after 32 layers of
// bf16 the gradients differed by as much as rounding noise does.)
#include "attention_common.cuh"

namespace {
using namespace attn;

struct LocalParams {
  AttnParams a;
  const int* items;      // [n][2]: first row, number of rows
};

// byte offset of element (row, col) of a [128 x 128] bf16 tile kept as two 64-column boxes
MMT_DEVICE uint32_t tile_offset(int row, int col) { return (uint32_t)(col >> 6) * CHUNK + sw128_offset(row, col & 63); }

constexpr int kLocalFwdThreads = 160;      // four softmax warps (one row per thread), one warp for TMA and MMA
constexpr size_t kLocalFwdSmem = 1024 + 6 * CHUNK + 5 * 8 + 16;

template <int DIM>
__global__ void __launch_bounds__(kLocalFwdThreads, 2)
attn_local_fwd_kernel(const __grid_constant__ CUtensorMap tm, const LocalParams lp) {
  const AttnParams& p = lp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + 2 * CHUNK;
  uint8_t* sV = sK + 2 * CHUNK;
  uint64_t* qk_full = reinterpret_cast<uint64_t*>(sV + 2 * CHUNK);
  uint64_t* v_full = qk_full + 1;
  uint64_t* s_full = qk_full + 2;
  uint64_t* p_full = qk_full + 3;
  uint64_t* o_full = qk_full + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(qk_full + 5);
  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm);
    mbar_init(qk_full, 1);
    mbar_init(v_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 4);
    mbar_init(o_full, 1);
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t t_s = warp_uniform(*tmem_slot), t_o = t_s + 128;      // S (P over its first 64 columns), O
  grid_dependency_sync();
  const int head = (int)blockIdx.x % p.n_q, item = (int)blockIdx.x / p.n_q;
  const int r0 = warp_uniform(lp.items[2 * item]), rows = lp.items[2 * item + 1];

  if (warp == 4) {
    const int kv_head = head / (p.n_q / p.n_kv);
    const int xq = head * DIM, xk = (p.n_q + kv_head) * DIM, xv = (p.n_q + p.n_kv + kv_head) * DIM;
    if (elect_one()) {
      mbar_expect_tx(qk_full, 4 * CHUNK);
      tma_load_2d(sQ, &tm, qk_full, xq, r0);
      tma_load_2d(sK, &tm, qk_full, xk, r0);
      tma_load_2d(sQ + CHUNK, &tm, qk_full, xq + 64, r0);
      tma_load_2d(sK + CHUNK, &tm, qk_full, xk + 64, r0);
      mbar_expect_tx(v_full, 2 * CHUNK);
      tma_load_2d(sV, &tm, v_full, xv, r0);
      tma_load_2d(sV + CHUNK, &tm, v_full, xv + 64, r0);
    }
    __syncwarp();
    if (mbar_wait_warp(qk_full, 0, p.ew, 800)) {
      const uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k)
          tc_mma_ss(t_s, desc_kmajor(smem_u32(sQ), k), desc_kmajor(smem_u32(sK), k), idesc_s, k != 0);
        tc_commit(s_full);
      }
      __syncwarp();
      if (mbar_wait_warp(v_full, 0, p.ew, 801) && mbar_wait_warp(p_full, 0, p.ew, 802)) {
        tc_fence_after();
        const uint32_t idesc_pv = make_idesc_bf16(BQ, DIM, 0, 1);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BKV / 16; ++k)
            tc_mma_ts(t_o, t_s + (uint32_t)(k * 8), desc_mnmajor(smem_u32(sV), k), idesc_pv, k != 0);
          tc_commit(o_full);
        }
      }
    }
    __syncwarp();
  } else {
    const int row = warp * 32 + lane;
    const int qrow = r0 + row;
    const bool row_ok = row < rows && qrow < p.T;
    int lo = 0, hi = 0;                          // visible columns of this row, relative to the pack
    if (row_ok) {
      lo = p.seq_lo[qrow];
      hi = p.seq_hi[qrow];
      if (p.causal) hi = min(hi, qrow + 1);
      lo -= r0;
      hi -= r0;
    }
    const float sl2 = p.scale * LOG2E;
    const float2 sl2_2 = make_float2(sl2, sl2);
    const uint32_t lane_addr = ((uint32_t)(warp * 32) << 16);
    bool ok = __all_sync(0xffffffffu, mbar_wait(s_full, 0, p.ew, 810));
    float m = -INFINITY, l = 0.f;
    if (ok) {
      tc_fence_after();
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + lane_addr + c * 32, r[c]);
      tmem_wait_ld();
      uint32_t vis[4];
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        vis[c] = visible_bits(lo - c * 32, hi - c * 32);
        if (__any_sync(0xffffffffu, vis[c] != 0u)) {
#pragma unroll
          for (int i = 0; i < 32; ++i) mx[c] = fmaxf(mx[c], (vis[c] >> i) & 1u ? __uint_as_float(r[c][i]) : -INFINITY);
        }
      }
      m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const float bias = m == -INFINITY ? 0.f : -m * sl2;
      const float2 bias2 = make_float2(bias, bias);
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
        // columns that no row of the warp sees (the other window of the pack) need no exponentials
        if (__any_sync(0xffffffffu, vis[c] != 0u)) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 t = fma2(make_float2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), sl2_2, bias2);
            float2 e = make_float2(exp2f(t.x), exp2f(t.y));
            if (!((vis[c] >> i) & 1u)) e.x = 0.f;
            if (!((vis[c] >> (i + 1)) & 1u)) e.y = 0.f;
            sum += e.x + e.y;
            pk[i >> 1] = pack_bf16x2(e.x, e.y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = 0u;
        }
        tmem_st_32x32b_x16(t_s + lane_addr + c * 16, pk);
      }
      l = sum;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      ok = __all_sync(0xffffffffu, mbar_wait(o_full, 0, p.ew, 811));
    }
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + (long)qrow * (p.n_q * DIM) + head * DIM;
      uint32_t o[DIM / 16][16];
#pragma unroll
      for (int c = 0; c < DIM / 16; ++c) tmem_ld_32x32b_x16(t_o + lane_addr + c * 16, o[c]);
      tmem_wait_ld();
      if (row_ok) {
#pragma unroll
        for (int c = 0; c < DIM / 16; ++c) {
          uint32_t v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            v[i] = pack_bf16x2(__uint_as_float(o[c][2 * i]) * inv, __uint_as_float(o[c][2 * i + 1]) * inv);
          *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<uint4*>(dst + c * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
        }
        p.lse[(long)head * p.T + qrow] = l > 0.f ? m * p.scale + logf(l) : INFINITY;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) tmem_dealloc(t_s, 256);
}

// Backward.  S = Q K^T and dP = dO V^T (query rows in the tensor-memory lanes); eight softmax warps (two per lane
// quadrant, 64 columns each) turn them into P and dS, bf16, in shared memory; then dV = P^T dO, dK = dS^T Q (A operands
// read MN-major) and dQ = dS K.  P takes the place of V, which is no longer needed.
// Tensor memory: S 0, dP 128, dQ 256, dK 384, dV over S.
constexpr int kLocalBwdThreads = 288;
constexpr size_t kLocalBwdSmem = 1024 + 10 * CHUNK + 2 * 128 * 4 + 7 * 8 + 16;

template <int DIM>
__global__ void __launch_bounds__(kLocalBwdThreads, 1)
attn_local_bwd_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                      const LocalParams lp) {
  const AttnParams& p = lp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + 2 * CHUNK;
  uint8_t* sDO = sK + 2 * CHUNK;
  uint8_t* sV = sDO + 2 * CHUNK;               // then P
  uint8_t* sDS = sV + 2 * CHUNK;
  float* sDelta = reinterpret_cast<float*>(sDS + 2 * CHUNK);      // [2 halves of the head's columns][128 rows]
  uint64_t* qk_full = reinterpret_cast<uint64_t*>(sDelta + 256);
  uint64_t* dov_full = qk_full + 1;
  uint64_t* s_full = qk_full + 2;
  uint64_t* pds_full = qk_full + 3;
  uint64_t* grad_full = qk_full + 4;           // [3]: dV, dK, dQ
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(qk_full + 7);
  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm);
    tma_prefetch_desc(&tm_do);
    mbar_init(qk_full, 1);
    mbar_init(dov_full, 1);
    mbar_init(s_full, 1);
    mbar_init(pds_full, 8);
    for (int i = 0; i < 3; ++i) mbar_init(&grad_full[i], 1);
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t t_s = warp_uniform(*tmem_slot), t_dp = t_s + 128, t_dq = t_s + 256, t_dk = t_s + 384, t_dv = t_s;
  grid_dependency_sync();
  const int head = (int)blockIdx.x % p.n_q, item = (int)blockIdx.x / p.n_q;
  const int r0 = warp_uniform(lp.items[2 * item]), rows = lp.items[2 * item + 1];
  const int xq = head * DIM, xk = (p.n_q + head) * DIM, xv = (2 * p.n_q + head) * DIM;

  if (warp == 8) {
    if (elect_one()) {
      mbar_expect_tx(qk_full, 4 * CHUNK);
      tma_load_2d(sQ, &tm, qk_full, xq, r0);
      tma_load_2d(sK, &tm, qk_full, xk, r0);
      tma_load_2d(sQ + CHUNK, &tm, qk_full, xq + 64, r0);
      tma_load_2d(sK + CHUNK, &tm, qk_full, xk + 64, r0);
      mbar_expect_tx(dov_full, 4 * CHUNK);
      tma_load_2d(sDO, &tm_do, dov_full, xq, r0);
      tma_load_2d(sV, &tm, dov_full, xv, r0);
      tma_load_2d(sDO + CHUNK, &tm_do, dov_full, xq + 64, r0);
      tma_load_2d(sV + CHUNK, &tm, dov_full, xv + 64, r0);
    }
    __syncwarp();
    const uint32_t q = smem_u32(sQ), k_ = smem_u32(sK), d_o = smem_u32(sDO), v = smem_u32(sV), ds = smem_u32(sDS);
    const uint32_t idesc_1 = make_idesc_bf16(128, 128, 0, 0);
    bool ok = mbar_wait_warp(qk_full, 0, p.ew, 820);
    if (ok) {
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k) tc_mma_ss(t_s, desc_kmajor(q, k), desc_kmajor(k_, k), idesc_1, k != 0);
      }
      __syncwarp();
      ok = mbar_wait_warp(dov_full, 0, p.ew, 821);
    }
    if (ok) {
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k) tc_mma_ss(t_dp, desc_kmajor(d_o, k), desc_kmajor(v, k), idesc_1, k != 0);
        tc_commit(s_full);
      }
      __syncwarp();
      ok = mbar_wait_warp(pds_full, 0, p.ew, 822);
    }
    if (ok) {
      tc_fence_after();
      const uint32_t idesc_t = make_idesc_bf16(128, DIM, 1, 1), idesc_q = make_idesc_bf16(128, DIM, 0, 1);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 8; ++k) tc_mma_ss(t_dv, desc_mnmajor(v, k), desc_mnmajor(d_o, k), idesc_t, k != 0);
        tc_commit(&grad_full[0]);
#pragma unroll
        for (int k = 0; k < 8; ++k) tc_mma_ss(t_dk, desc_mnmajor(ds, k), desc_mnmajor(q, k), idesc_t, k != 0);
        tc_commit(&grad_full[1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) tc_mma_ss(t_dq, desc_kmajor(ds, k), desc_mnmajor(k_, k), idesc_q, k != 0);
        tc_commit(&grad_full[2]);
      }
      __syncwarp();
    }
  } else {
    const int q4 = warp & 3, half = warp >> 2;
    const int row = q4 * 32 + lane;
    const int grow = r0 + row;
    const bool row_ok = row < rows && grow < p.T;
    const uint32_t lane_addr = ((uint32_t)(q4 * 32) << 16);
    int lo = 0, hi = 0;
    float lse_l2 = 0.f, part = 0.f;
    if (row_ok) {
      lo = p.seq_lo[grow];
      hi = p.seq_hi[grow];
      if (p.causal) hi = min(hi, grow + 1);
      lo -= r0;
      hi -= r0;
      lse_l2 = p.lse[(long)head * p.T + grow] * LOG2E;
      // delta = sum of out * dout in the order in which a warp with a pair of columns per lane adds it up (the lane's
      // pairs, then lanes 16, 8, 4, 2 and 1 apart), so that it has the same bits as attn_delta_kernel's; this thread has
      // the even or the odd lanes, and the last step joins the two
      const long at = (long)grow * (p.n_q * DIM) + head * DIM;
      float lane_sum[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) lane_sum[i] = 0.f;
#pragma unroll
      for (int i = 0; i < DIM / 8; ++i) {
        const uint4 o = *reinterpret_cast<const uint4*>(p.out + at + i * 8);
        const uint4 d = *reinterpret_cast<const uint4*>(p.dout + at + i * 8);
        const uint32_t ow[2] = {half ? o.y : o.x, half ? o.w : o.z}, dw[2] = {half ? d.y : d.x, half ? d.w : d.z};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 a = unpack_bf16x2(ow[j]), b = unpack_bf16x2(dw[j]);
          lane_sum[(2 * i + j) & 15] += a.x * b.x + a.y * b.y;
        }
      }
#pragma unroll
      for (int step = 8; step > 0; step >>= 1)
#pragma unroll
        for (int i = 0; i < step; ++i) lane_sum[i] += lane_sum[i + step];
      part = lane_sum[0];
    }
    sDelta[half * 128 + row] = part;
    quadrant_bar_sync<2>(q4);
    const float delta = part + sDelta[(half ^ 1) * 128 + row];
    const float sl2 = p.scale * LOG2E;
    const float2 sl2_2 = make_float2(sl2, sl2), scale_2 = make_float2(p.scale, p.scale);
    const float2 lse_2 = make_float2(-lse_l2, -lse_l2), delta_2 = make_float2(-delta, -delta);
    bool ok = __all_sync(0xffffffffu, mbar_wait(s_full, 0, p.ew, 830));
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int col0 = half * 64 + c * 32;
        uint32_t r_s[32], r_dp[32];
        tmem_ld_32x32b_x32(t_s + lane_addr + (uint32_t)col0, r_s);
        tmem_ld_32x32b_x32(t_dp + lane_addr + (uint32_t)col0, r_dp);
        const uint32_t vis = visible_bits(lo - col0, hi - col0);
        tmem_wait_ld();
        uint32_t pk_p[16], pk_ds[16];
        if (__any_sync(0xffffffffu, vis != 0u)) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float2 e = fma2(make_float2(__uint_as_float(r_s[i]), __uint_as_float(r_s[i + 1])), sl2_2, lse_2);
            e = make_float2(exp2f(e.x), exp2f(e.y));
            if (!((vis >> i) & 1u)) e.x = 0.f;
            if (!((vis >> (i + 1)) & 1u)) e.y = 0.f;
            float2 d = add2(make_float2(__uint_as_float(r_dp[i]), __uint_as_float(r_dp[i + 1])), delta_2);
            d = mul2(mul2(e, d), scale_2);
            pk_p[i >> 1] = pack_bf16x2(e.x, e.y);
            pk_ds[i >> 1] = pack_bf16x2(d.x, d.y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) pk_p[i] = pk_ds[i] = 0u;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t at = tile_offset(row, col0 + g * 8);
          *reinterpret_cast<uint4*>(sV + at) = make_uint4(pk_p[g * 4], pk_p[g * 4 + 1], pk_p[g * 4 + 2], pk_p[g * 4 + 3]);
          *reinterpret_cast<uint4*>(sDS + at) =
              make_uint4(pk_ds[g * 4], pk_ds[g * 4 + 1], pk_ds[g * 4 + 2], pk_ds[g * 4 + 3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
    }
    // gradients: the two warps of a lane quadrant share a row's columns in chunks of 16
#pragma unroll 1
    for (int t = 0; t < 3 && ok; ++t) {
      ok = __all_sync(0xffffffffu, mbar_wait(&grad_full[t], 0, p.ew, 831));
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = (t == 0 ? t_dv : (t == 1 ? t_dk : t_dq)) + lane_addr;
      __nv_bfloat16* dst = p.dqkv + (long)grow * p.ld + (t == 0 ? xv : (t == 1 ? xk : xq));
#pragma unroll
      for (int c0 = 0; c0 < DIM / 16; c0 += 2) {
        const int c = c0 + half;
        if (c < DIM / 16) {
          uint32_t r[16];
          tmem_ld_32x32b_x16(acc + (uint32_t)(c * 16), r);
          tmem_wait_ld();
          if (row_ok) {
            uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<uint4*>(dst + c * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(t_s, 512);
}

template <int DIM>
int launch_local_fwd(const CUtensorMap& tm, const LocalParams& lp, int n_items, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_local_fwd_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kLocalFwdSmem);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  return (int)launch_dependent(attn_local_fwd_kernel<DIM>, (unsigned)n_items * lp.a.n_q, kLocalFwdThreads, kLocalFwdSmem,
                               st, tm, lp);
}

template <int DIM>
int launch_local_bwd(const CUtensorMap& tm, const CUtensorMap& tdo, const LocalParams& lp, int n_items, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_local_bwd_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kLocalBwdSmem);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  return (int)launch_dependent(attn_local_bwd_kernel<DIM>, (unsigned)n_items * lp.a.n_q, kLocalBwdThreads, kLocalBwdSmem,
                               st, tm, tdo, lp);
}

LocalParams local_params(const void* qkv, const int* seq_lo, const int* seq_hi, const int* items, long T, int n_q,
                         int n_kv, int dim, long ld, int causal, float scale) {
  LocalParams lp = {};
  lp.a.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  lp.a.seq_lo = seq_lo;
  lp.a.seq_hi = seq_hi;
  lp.a.T = (int)T; lp.a.n_q = n_q; lp.a.n_kv = n_kv; lp.a.dim = dim; lp.a.ld = ld;
  lp.a.causal = causal; lp.a.scale = scale;
  lp.a.ew = mmt_error_word();
  lp.items = items;
  return lp;
}

}  // namespace

// As mmt_attn_fwd for sequences of at most 128 rows; `items` lists packs of whole sequences (device, [n_items][2]).
extern "C" int mmt_attn_local_fwd(const void* qkv, void* out, float* lse, const int* seq_lo, const int* seq_hi,
                                  const int* items, int n_items, long T, int n_q, int n_kv, int dim, long ld, int causal,
                                  float scale, void* stream) {
  if (T <= 0 || n_items <= 0) return 0;
  if (mmt_ensure_context(qkv)) return -7;
  if ((dim != 80 && dim != 128) || n_q % n_kv || (ld & 7)) return -2;
  CUtensorMap tm;
  const int r = mmt_make_tmap_2d(&tm, qkv, (uint64_t)(n_q + 2 * n_kv) * dim, (uint64_t)T, (uint64_t)ld, 64, 128);
  if (r) return 1000 + r;
  LocalParams lp = local_params(qkv, seq_lo, seq_hi, items, T, n_q, n_kv, dim, ld, causal, scale);
  lp.a.out = reinterpret_cast<__nv_bfloat16*>(out);
  lp.a.lse = lse;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return dim == 80 ? launch_local_fwd<80>(tm, lp, n_items, st) : launch_local_fwd<128>(tm, lp, n_items, st);
}

// As mmt_attn_bwd for sequences of at most 128 rows and n_q == n_kv; needs no delta and no workspace.
extern "C" int mmt_attn_local_bwd(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv,
                                  const int* seq_lo, const int* seq_hi, const int* items, int n_items, long T, int n_q,
                                  int n_kv, int dim, long ld, int causal, float scale, void* stream) {
  if (T <= 0 || n_items <= 0) return 0;
  if (mmt_ensure_context(qkv)) return -7;
  if ((dim != 80 && dim != 128) || n_q != n_kv || (ld & 7)) return -2;
  CUtensorMap tm, tdo;
  int r = mmt_make_tmap_2d(&tm, qkv, (uint64_t)(n_q + 2 * n_kv) * dim, (uint64_t)T, (uint64_t)ld, 64, 128);
  if (r) return 1000 + r;
  r = mmt_make_tmap_2d(&tdo, dout, (uint64_t)n_q * dim, (uint64_t)T, (uint64_t)n_q * dim, 64, 128);
  if (r) return 2000 + r;
  LocalParams lp = local_params(qkv, seq_lo, seq_hi, items, T, n_q, n_kv, dim, ld, causal, scale);
  lp.a.out = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(out));
  lp.a.lse = const_cast<float*>(lse);
  lp.a.dout = reinterpret_cast<const __nv_bfloat16*>(dout);
  lp.a.dqkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return dim == 80 ? launch_local_bwd<80>(tm, tdo, lp, n_items, st) : launch_local_bwd<128>(tm, tdo, lp, n_items, st);
}
