// One tile per CTA for grids of less than one wave; included by gemm.cu (same parameters, operand layouts and ring).
//
// A small output (256 rows of activations) has 10 to 80 tiles for 148 SMs, and its time is one tile's chain of k-blocks.
// The persistent kernel's loops step through tiles and look at collective roles, and its narrow tiles took 0.235 us per
// k-block; here a 64-column tile takes 0.177 us.  The products and their order are those of the persistent kernel, and
// so are the bits.  (K shared by a cluster of CTAs, with the partial sums exchanged through distributed shared memory,
// was twice as fast again for long K, but adds in another order; see small_tile in gemm.cu.)
// Measured: 256 x 1280 x 3424 16.4 (persistent, 64 columns) -> 12.6 us, 256 x 3840 x 1280 9.2 -> 7.4 us.

// Arithmetic and store of eight finished columns of one row.
MMT_DEVICE void finish8(const GemmParams& p, long row, int col, float (&v)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] *= p.alpha;
  auto add8 = [&](const __nv_bfloat16* src) {
    const uint4 u = *reinterpret_cast<const uint4*>(src);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(w[j]);
      v[2 * j] += f.x;
      v[2 * j + 1] += f.y;
    }
  };
  if (p.bias) add8(p.bias + col);
  if (p.act == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = gelu_erf(v[j]);
  }
  if (p.residual) add8(p.residual + row * p.ldr + col);
  if (p.out_f32) {
    float* dst = reinterpret_cast<float*>(p.C) + row * p.ldc + col;
    if (p.accumulate) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += dst[j];
    }
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col;
    if (p.accumulate) add8(dst);
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                                pack_bf16x2(v[6], v[7]));
  }
}

constexpr int kSmallThreads = 64 + kEpiWarps * 32;

template <int BN>
struct SmallCfg {
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + BN * BK * 2;
  static constexpr int kStages = (int)((224u * 1024u) / STAGE_BYTES) > 8 ? 8 : (int)((224u * 1024u) / STAGE_BYTES);
  static constexpr uint32_t TMEM_COLS = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);
  static constexpr size_t SMEM = 1024 + (size_t)kStages * STAGE_BYTES + (2 * kStages + 1) * 8 + 16;
};

template <int BN>
__global__ void __launch_bounds__(kSmallThreads, 1)
gemm_bf16_small(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  using C_ = SmallCfg<BN>;
  constexpr int kStages = C_::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * C_::STAGE_BYTES);
  uint64_t* empty = full + kStages;
  uint64_t* tfull = empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int tiles_m = (p.M + BM - 1) / BM;
  const int tm = (int)blockIdx.x % tiles_m, tn = (int)blockIdx.x / tiles_m;
  const int KB = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C_::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t acc = warp_uniform(*tmem_slot);
  grid_dependency_wait();

  if (warp == 0) {
    int s = 0;
    uint32_t ph = 0;
    for (int kb = 0; kb < KB; ++kb) {
      if (!mbar_wait_warp(&empty[s], ph ^ 1, p.ew, 130)) break;
      uint8_t* sA = smem + (size_t)s * C_::STAGE_BYTES;
      uint8_t* sB = sA + C_::A_BYTES;
      if (elect_one()) {
        mbar_expect_tx(&full[s], C_::STAGE_BYTES);
        if (!p.a_mn) {
          tma_load_2d(sA, &tmA, &full[s], kb * BK, tm * BM);
        } else {
#pragma unroll
          for (int c = 0; c < BM / 64; ++c) tma_load_2d(sA + c * 8192, &tmA, &full[s], tm * BM + c * 64, kb * BK);
        }
        if (!p.b_mn) {
          tma_load_2d(sB, &tmB, &full[s], kb * BK, tn * BN);
        } else {
#pragma unroll
          for (int c = 0; c < BN / 64; ++c) tma_load_2d(sB + c * 8192, &tmB, &full[s], tn * BN + c * 64, kb * BK);
        }
      }
      __syncwarp();
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
    grid_dependents_launch();
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc_bf16(BM, BN, p.a_mn, p.b_mn);
    const uint32_t a_hi = smem_desc_hi(p.a_mn ? p.mn_sbo : 1024u), b_hi = smem_desc_hi(p.b_mn ? p.mn_sbo : 1024u);
    const uint32_t a_lo0 = smem_desc_lo(smem_u32(smem), p.a_mn ? p.mn_lbo : 16u);
    const uint32_t b_lo0 = smem_desc_lo(smem_u32(smem) + C_::A_BYTES, p.b_mn ? p.mn_lbo : 16u);
    const uint32_t a_k = (p.a_mn ? p.mn_kstep : (uint32_t)(UMMA_K * 2)) >> 4;
    const uint32_t b_k = (p.b_mn ? p.mn_kstep : (uint32_t)(UMMA_K * 2)) >> 4;
    int s = 0;
    uint32_t ph = 0;
    for (int kb = 0; kb < KB; ++kb) {
      if (!mbar_wait_warp(&full[s], ph, p.ew, 230)) break;
      const uint32_t so = (uint32_t)s * (C_::STAGE_BYTES >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          tc_mma_ss(acc, smem_desc_join(a_hi, a_lo0 + so + (uint32_t)k * a_k),
                    smem_desc_join(b_hi, b_lo0 + so + (uint32_t)k * b_k), idesc, (kb | k) != 0 ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
    if (elect_one()) tc_commit(tfull);
    __syncwarp();
  } else if (__all_sync(0xffffffffu, mbar_wait(tfull, 0, p.ew, 330))) {
    tc_fence_after();
    const int q = warp & 3, half = (warp - 2) >> 2;      // lane quadrant; even or odd chunks of 16 columns
    const int row = q * 32 + lane;
    const long grow = (long)tm * BM + row;
#pragma unroll
    for (int cc = 0; cc < BN / 32; ++cc) {
      const int ch = 2 * cc + half;
      uint32_t r[16];
      tmem_ld_32x32b_x16(acc + ((uint32_t)(q * 32) << 16) + (uint32_t)(ch * 16), r);
      tmem_wait_ld();
      if (grow < p.M) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = tn * BN + ch * 16 + h * 8;
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[h * 8 + i]);
          if (col < p.N) finish8(p, grow, col, v);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(acc, C_::TMEM_COLS);
}

template <int BN>
int launch_small(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t st) {
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_small<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)SmallCfg<BN>::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  return (int)launch_dependent(gemm_bf16_small<BN>, tiles, kSmallThreads, SmallCfg<BN>::SMEM, st, ta, tb, p);
}
