// Packed variable-length flash attention on tcgen05 (sm_100a), forward and backward.
//
// Layout.  One fused activation buffer qkv[T, ld] (bf16): q heads, then k heads, then v heads,
// `dim` columns each (dim = 80 for the vision encoder, 128 for the text decoder).  Sequences are
// packed along T; per-token arrays seq_lo[t], seq_hi[t] give the row range of the token's own
// sequence, which expresses window attention, whole-image attention and packed causal text with
// one mechanism: a query tile of 128 consecutive rows may span several (short) sequences and the
// mask keeps every row inside its own.  GQA: q head h reads kv head h / (n_q / n_kv).
//
// Forward: one CTA per pair of neighbouring 128-row query tiles of a q head, 10 warps (two softmax warp groups, a TMA
// producer, an MMA issuer); see the comment at attn_fwd2_kernel.
// head_dim 80 is not a multiple of the 64-column swizzle atom: every operand tile is fetched as two
// 64-column boxes (columns 0-63 and 64-127 of the head; the tail of the second box belongs to the
// next head or is zero fill and is never read).  As a K-major operand the fifth K=16 step reads the
// first 16 columns of the second box; as an MN-major operand N=80 covers box 0 and a quarter of
// box 1.  So there are no padded FLOPs and a single swizzle mode.
//
// Backward is two kernels without atomics: dK/dV (one CTA per KV tile, looping over the query
// tiles and the q heads of the group, accumulating in tensor memory) and dQ (one CTA per query
// tile, looping over KV tiles).  Both recompute P from the saved log-sum-exp.
//
// Replaces flash-attn's flash_attn_varlen_func reached through HF in the reference
// (python/models/qwen2_5_vl/modeling_qwen2_5_vl.py:431-448,540-557,694-711,1266-1281).
#include "attention_common.cuh"

namespace {
using namespace attn;

// ------------------------------------------------------------------------------------------------
// Forward: two neighbouring query tiles of one head per CTA, worked in ping-pong.
//
// With one tile per CTA the softmax warps are the limit: while they convert S of tile j the tensor core idles.  Here a
// CTA owns two query tiles, each with its own softmax warp group (4 warps, one query row per thread) and its own
// tensor-memory columns, while ONE TMA warp and ONE MMA warp serve both, so the tensor core computes S or PV of one
// tile while the other tile's rows are in the exponentials.
//   * Both tiles read the same K and V blocks (a two-stage ring): half the operand traffic of two independent tiles.
//     A tile skips the blocks outside its own visible range (packed sequences, causal).
//   * P never touches shared memory: the softmax threads write it as packed bf16 pairs over the first 64
//     columns of the S tile they have just read (tcgen05.st), and PV takes it as the tensor-memory A operand.
//   * A thread reads its 128 scores into registers once (the last 32 twice) and maximum, exponentials and sum run from
//     there, the scaling on packed fp32 pairs: per 128 x 128 tile the exponentials alone need 1024 cycles of an SM (16 per cycle), the MMAs
//     640 (head_dim 80), so everything else has to fit beside them.  Reading
//     the scores twice, one wait per 32 columns: 2.00 ms for one image of 16384 patches (16 heads of 80), now 1.59 ms.
//   * O stays in tensor memory for the whole KV loop (PV accumulates).  The running maximum is lazy: O and l
//     are rescaled only when a row's maximum grew by more than 2^8 since the value in use, which after the
//     first tiles is rare; the rescale is a tensor-memory read-modify-write by the row's own thread, safe
//     because S of tile j is only published after PV of tile j-1 has completed.
//   * KV tiles that are entirely visible to every row of a warp skip the per-element mask.
// Tensor memory: S/P of tile w at columns [128w, 128w+128), O of tile w at [256+128w, 256+128w+DIM).
// Shared memory: Q of each tile and two stages of K and V, 32 KB each (two 64-column boxes).
// ------------------------------------------------------------------------------------------------
constexpr int kFwd2Threads = 320;

template <int DIM>
__global__ void __launch_bounds__(kFwd2Threads, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tm, const AttnParams p, const int n_pairs) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                         // [tile][2 boxes]
  uint8_t* sK = sQ + 4 * CHUNK;               // [stage][2 boxes]
  uint8_t* sV = sK + 4 * CHUNK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 4 * CHUNK);
  uint64_t* q_full = bars;          // [2] per tile
  uint64_t* k_full = bars + 2;      // [2] per stage
  uint64_t* k_empty = bars + 4;     // [2] per stage
  uint64_t* v_full = bars + 6;      // [2] per stage
  uint64_t* v_empty = bars + 8;     // [2] per stage
  uint64_t* s_full = bars + 10;     // [2] per tile
  uint64_t* p_full = bars + 12;     // [2] per tile
  uint64_t* pv_done = bars + 14;    // [2] per tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  constexpr int X2 = 64;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  grid_dependency_sync();
  // non-causal: the CTAs that run together share a head, so its K and V stay in L2 however long the sequence;
  // causal: the last query tiles see the most KV blocks and are started first, over all heads (longest work first)
  const int head = p.causal ? (int)blockIdx.x % p.n_q : (int)blockIdx.x / n_pairs;
  const int pair = p.causal ? n_pairs - 1 - (int)blockIdx.x / p.n_q : (int)blockIdx.x % n_pairs;
  const int kv_head = head / (p.n_q / p.n_kv);
  const int xq = head * DIM, xk = (p.n_q + kv_head) * DIM, xv = (p.n_q + p.n_kv + kv_head) * DIM;
  // The CTA walks blocks of 128 KV rows; block j is worked on by tile w if first[w] <= j < last[w].  Tiles of one sequence
  // start at the same row and share their blocks.  If the second tile starts in another sequence, its blocks follow those
  // of the first one and are counted from its own first row: a tile's blocks, and with them its sums, do not depend on
  // its neighbour.
  int q0[2], first[2], last[2], lo_w[2] = {0, 0};
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    q0[w] = (pair * 2 + w) * BQ;
    first[w] = last[w] = 0;
    if (q0[w] < p.T) {
      const int q_last = min(q0[w] + BQ, p.T) - 1;
      lo_w[w] = p.seq_lo[q0[w]];
      const int hi = p.causal ? min(p.seq_hi[q_last], q_last + 1) : p.seq_hi[q_last];
      if (w == 1 && lo_w[1] != lo_w[0]) first[1] = last[0];
      last[w] = first[w] + (hi - lo_w[w] + BKV - 1) / BKV;
    }
    first[w] = warp_uniform(first[w]);
    last[w] = warp_uniform(last[w]);
    lo_w[w] = warp_uniform(lo_w[w]);
  }
  const int own1 = first[1] > 0 ? first[1] : 0x7fffffff;        // first block that is counted from tile 1's first row
  auto block_row = [&](int j) { return j < own1 ? lo_w[0] + j * BKV : lo_w[1] + (j - own1) * BKV; };
  const int n_blocks = max(last[0], last[1]);

  if (warp == 8) {
    // ------------------------------ TMA producer ------------------------------
    auto load = [&](uint8_t* dst, uint64_t* bar, int x, int y) {
      if (elect_one()) {
        mbar_expect_tx(bar, 2 * CHUNK);
        tma_load_2d(dst, &tm, bar, x, y);
        tma_load_2d(dst + CHUNK, &tm, bar, x + X2, y);
      }
      __syncwarp();
    };
    if (last[0] > first[0]) load(sQ, &q_full[0], xq, q0[0]);
    for (int j = 0; j < n_blocks; ++j) {
      const int st = j & 1;
      const uint32_t free_parity = (uint32_t)(((j >> 1) & 1) ^ 1);
      const int r0 = block_row(j);
      if (!mbar_wait_warp(&k_empty[st], free_parity, p.ew, 410)) break;
      load(sK + st * 2 * CHUNK, &k_full[st], xk, r0);
      if (j == 0 && last[1] > first[1]) load(sQ + 2 * CHUNK, &q_full[1], xq, q0[1]);
      if (!mbar_wait_warp(&v_empty[st], free_parity, p.ew, 411)) break;
      load(sV + st * 2 * CHUNK, &v_full[st], xv, r0);
    }
  } else if (warp == 9) {
    // ------------------------------ MMA issuer ------------------------------
    {
      const uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);
      const uint32_t idesc_pv = make_idesc_bf16(BQ, DIM, 0, 1);
      const uint32_t hi = smem_desc_hi(1024);
      const uint32_t q_lo = smem_desc_lo(smem_u32(sQ), 16);
      const uint32_t k_lo = smem_desc_lo(smem_u32(sK), 16);
      const uint32_t v_lo = smem_desc_lo(smem_u32(sV), CHUNK);
      constexpr uint32_t kPair = (2 * CHUNK) >> 4;      // one tile's or stage's two boxes
      auto issue_s = [&](int w, int j) {
        const uint32_t d = tmem_base + (uint32_t)(w * 128);
        const uint32_t a = q_lo + (uint32_t)w * kPair, b = k_lo + (uint32_t)(j & 1) * kPair;
        if (!elect_one()) return;
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k) {
          const uint32_t off = (uint32_t)(((k >> 2) * CHUNK + (k & 3) * 32) >> 4);
          tc_mma_ss(d, smem_desc_join(hi, a + off), smem_desc_join(hi, b + off), idesc_s, k != 0);
        }
        tc_commit(&s_full[w]);
      };
      auto sees = [&](int w, int j) { return j >= first[w] && j < last[w]; };
      int seen[2] = {0, 0};                             // blocks of tile w whose P has been consumed
      bool ok = true;
      if (n_blocks > 0) ok = mbar_wait_warp(&k_full[0], 0, p.ew, 511);
      for (int w = 0; w < 2 && ok; ++w) {
        if (!sees(w, 0)) continue;
        ok = mbar_wait_warp(&q_full[w], 0, p.ew, 510);
        if (ok) issue_s(w, 0);
        __syncwarp();
      }
      if (ok && n_blocks > 0 && elect_one()) tc_commit(&k_empty[0]);
      for (int j = 0; j < n_blocks && ok; ++j) {
        const int nx = j + 1;
        bool have_k = false, have_v = false;
        for (int w = 0; w < 2 && ok; ++w) {
          if (sees(w, j)) {
            if (!have_v && !mbar_wait_warp(&v_full[j & 1], (j >> 1) & 1, p.ew, 513)) { ok = false; break; }
            have_v = true;
            if (!mbar_wait_warp(&p_full[w], seen[w] & 1, p.ew, 512)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d = tmem_base + 256u + (uint32_t)(w * 128);
            const uint32_t a = tmem_base + (uint32_t)(w * 128);
            const uint32_t b = v_lo + (uint32_t)(j & 1) * kPair;
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < BKV / 16; ++k)
                tc_mma_ts(d, a + (uint32_t)(k * 8), smem_desc_join(hi, b + (uint32_t)(k * (2048 >> 4))), idesc_pv,
                          (seen[w] | k) != 0);
              if (j == last[w] - 1) tc_commit(&pv_done[w]);
            }
            __syncwarp();
            ++seen[w];
          }
          if (w == 1 && elect_one()) tc_commit(&v_empty[j & 1]);
          __syncwarp();
          if (sees(w, nx)) {
            if (!have_k && !mbar_wait_warp(&k_full[nx & 1], (nx >> 1) & 1, p.ew, 514)) { ok = false; break; }
            have_k = true;
            if (nx == first[w] && !mbar_wait_warp(&q_full[w], 0, p.ew, 515)) { ok = false; break; }
            issue_s(w, nx);
            __syncwarp();
          }
        }
        if (ok && nx < n_blocks && elect_one()) tc_commit(&k_empty[nx & 1]);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ softmax + epilogue, one warp group per tile ------------------------------
    const int w = warp >> 2;             // tile
    const int q = warp & 3;              // tensor-memory lane quadrant of this warp
    const int j0 = first[w], j1 = last[w];
    if (j1 > j0) {
      const int row = q * 32 + lane;
      const int qrow = q0[w] + row;
      const bool row_ok = qrow < p.T;
      const int lo = row_ok ? p.seq_lo[qrow] : 0;
      int hi = row_ok ? p.seq_hi[qrow] : 0;
      if (p.causal) hi = min(hi, qrow + 1);
      const float sl2 = p.scale * LOG2E;
      const float2 sl2_2 = make_float2(sl2, sl2);
      const uint32_t lane_addr = ((uint32_t)(q * 32) << 16);
      const uint32_t s_addr = tmem_base + lane_addr + (uint32_t)(w * 128);
      const uint32_t o_addr = tmem_base + lane_addr + 256u + (uint32_t)(w * 128);
      float m_ref = -INFINITY, l = 0.f;
      bool ok = true;
      for (int j = j0; j < j1; ++j) {
        const int kv0 = block_row(j);
        ok = __all_sync(0xffffffffu, mbar_wait(&s_full[w], (j - j0) & 1, p.ew, 610));
        if (!ok) break;
        tc_fence_after();
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, r[c]);
        const bool full = __all_sync(0xffffffffu, kv0 >= lo && kv0 + BKV <= hi);
        tmem_wait_ld();
        // row maximum over the visible columns
        uint32_t vis[4];
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (full) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2)
              mx4[c] = max3(mx4[c], __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            vis[c] = visible_bits(lo - (kv0 + c * 32), hi - (kv0 + c * 32));
#pragma unroll
            for (int i = 0; i < 32; ++i)
              mx4[c] = fmaxf(mx4[c], (vis[c] >> i) & 1u ? __uint_as_float(r[c][i]) : -INFINITY);
          }
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // lazy running maximum: adopt a new reference only when it moved by more than 2^8
        const float m_new = fmaxf(m_ref, mx);
        const bool need = (m_new - m_ref) * sl2 > 8.f;        // false when both are -inf (NaN compares false)
        if (j == j0) {
          if (need) m_ref = m_new;                             // O does not exist yet: nothing to rescale
        } else if (__any_sync(0xffffffffu, need)) {
          const float alpha = need ? exp2f((m_ref - m_new) * sl2) : 1.f;   // exp2(-inf) = 0 for a row without history
          l *= alpha;
          if (need) m_ref = m_new;
#pragma unroll 1
          for (int c = 0; c < DIM / 16; ++c) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_addr + c * 16, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c * 16, o);
          }
        }
        const float bias = (m_ref == -INFINITY) ? 0.f : -m_ref * sl2;
        const float2 bias2 = make_float2(bias, bias);
        // P = exp2(S * sl2 + bias) as bf16 pairs, written over the columns of S
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // the last 32 scores are read a second time instead of being held over the first 96: they and the packed
          // results would not fit the register file together
          if (c == 1) tmem_ld_32x32b_x32(s_addr + 96, r[3]);
          if (c == 3) tmem_wait_ld();
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 t = fma2(make_float2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), sl2_2, bias2);
            float2 e = make_float2(exp2f(t.x), exp2f(t.y));
            if (!full) {
              if (!((vis[c] >> i) & 1u)) e.x = 0.f;
              if (!((vis[c] >> (i + 1)) & 1u)) e.y = 0.f;
            }
            sum += e.x + e.y;
            pk[i >> 1] = pack_bf16x2(e.x, e.y);
          }
          tmem_st_32x32b_x16(s_addr + c * 16, pk);
        }
        l += sum;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[w]);
      }
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[w], 0, p.ew, 611));
      if (ok) {
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
        __nv_bfloat16* dst = p.out + (long)qrow * (p.n_q * DIM) + head * DIM;
#pragma unroll
        for (int c = 0; c < DIM / 16; ++c) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(o_addr + c * 16, o);
          tmem_wait_ld();
          if (row_ok) {
            uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
              v[i] = pack_bf16x2(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<uint4*>(dst + c * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
          }
        }
        if (row_ok) p.lse[(long)head * p.T + qrow] = l > 0.f ? m_ref * p.scale + logf(l) : INFINITY;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem_base, 512);
}

constexpr size_t kFwdSmem = 1024 + 12 * CHUNK + 17 * 8 + 16;

template <int DIM>
int launch_fwd2(const CUtensorMap& tm, const AttnParams& p, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd2_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kFwdSmem);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  const int n_pairs = ((p.T + BQ - 1) / BQ + 1) / 2;
  launch_dependent(attn_fwd2_kernel<DIM>, n_pairs * p.n_q, kFwd2Threads, kFwdSmem, st, tm, p, n_pairs);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" int mmt_attn_fwd(const void* qkv, void* out, float* lse, const int* seq_lo, const int* seq_hi, long T,
                            int n_q, int n_kv, int dim, long ld, int causal, float scale, void* stream) {
  if (T <= 0) return 0;
  if (mmt_ensure_context(qkv)) return -7;
  if ((dim != 80 && dim != 128) || n_q % n_kv || (ld & 7)) return -2;
  CUtensorMap tm;
  const uint64_t width = (uint64_t)(n_q + 2 * n_kv) * dim;
  int r = mmt_make_tmap_2d(&tm, qkv, width, (uint64_t)T, (uint64_t)ld, 64, 128);
  if (r) return 1000 + r;
  AttnParams p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.seq_lo = seq_lo;
  p.seq_hi = seq_hi;
  p.T = (int)T; p.n_q = n_q; p.n_kv = n_kv; p.dim = dim; p.ld = ld;
  p.causal = causal; p.scale = scale;
  p.ew = mmt_error_word();
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return dim == 80 ? launch_fwd2<80>(tm, p, st) : launch_fwd2<128>(tm, p, st);
}
