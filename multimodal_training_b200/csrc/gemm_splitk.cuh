// Split-K GEMM for grids that leave most SMs idle; included by gemm.cu (same parameters, operand layouts and ring).
//
// The gradient of a square projection has 25 to 70 tiles for 148 SMs, and
// one SM takes operands in at about 100 GB/s whatever the tile: the GEMM's time is then its longest K loop.  Here a
// cluster of S CTAs shares one 128 x BN tile: CTA r multiplies the r-th part of K, then every CTA owns BN / S of the
// tile's columns, receives the other CTAs' fp32 partial sums of those columns in its (by then idle) operand ring through
// distributed shared memory, adds them in rank order and finishes the columns.  The reduction is spread over all S CTAs,
// needs no workspace, no flags and no second launch, and its result does not depend on timing.
// Measured: weight gradient 1280 x 1280 x 4096 25.8 (unsplit) -> 17.6 us as 70 tiles of 192 columns over 2 CTAs; the
// exchange costs 1 to 6 us, growing with the tile, so wide tiles are split for long K only (small_tile in gemm.cu).

MMT_DEVICE void st_cluster_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

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

constexpr int kSplitThreads = 64 + kEpiWarps * 32;

template <int BN>
struct SplitCfg {
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + BN * BK * 2;
  static constexpr int kStages = (int)((224u * 1024u) / STAGE_BYTES) > 8 ? 8 : (int)((224u * 1024u) / STAGE_BYTES);
  static constexpr uint32_t TMEM_COLS = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);
  static constexpr size_t SMEM = 1024 + (size_t)kStages * STAGE_BYTES + (2 * kStages + 1) * 8 + 16;
  static_assert(128 * BN * 4 <= kStages * (int)STAGE_BYTES, "the partial sums fit the idle ring");
};

template <int BN, int S>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_bf16_splitk(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  using C_ = SplitCfg<BN>;
  constexpr int kStages = C_::kStages;
  constexpr int W = BN / S;                       // columns that one CTA finishes
  static_assert(W % 16 == 0, "column chunks of 16 have one owner");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * C_::STAGE_BYTES);
  uint64_t* empty = full + kStages;
  uint64_t* tfull = empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  const int warp = warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int tiles_m = (p.M + BM - 1) / BM;
  const int tile = (int)blockIdx.x / S;
  const int tm = tile % tiles_m, tn = tile / tiles_m;
  const int KB = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long)KB * rank / S), kb1 = (int)((long)KB * (rank + 1) / S);

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

  bool ok = true;
  if (warp == 0) {
    int s = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
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
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full[s], ph, p.ew, 230)) break;
      const uint32_t so = (uint32_t)s * (C_::STAGE_BYTES >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          tc_mma_ss(acc, smem_desc_join(a_hi, a_lo0 + so + (uint32_t)k * a_k),
                    smem_desc_join(b_hi, b_lo0 + so + (uint32_t)k * b_k), idesc, (kb > kb0 || k != 0) ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
    if (elect_one()) tc_commit(tfull);
    __syncwarp();
  } else {
    ok = __all_sync(0xffffffffu, mbar_wait(tfull, 0, p.ew, 330));
    tc_fence_after();
  }
  // every CTA's MMAs have read their operands: the rings may take partial sums.  (All threads of all CTAs pass both
  // cluster barriers, also after a wait that ran out.)
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const int q = warp & 3, half = (warp - 2) >> 2;
  const int row = q * 32 + lane;
  const uint32_t taddr = acc + ((uint32_t)(q * 32) << 16);
  if (warp >= 2 && ok) {
#pragma unroll
    for (int ch = 0; ch < BN / 16; ++ch) {
      const int owner = ch * 16 / W;
      if ((ch & 1) != half || owner == rank) continue;
      uint32_t r[16];
      tmem_ld_32x32b_x16(taddr + (uint32_t)(ch * 16), r);
      tmem_wait_ld();
      const int slot = rank < owner ? rank : rank - 1;
      const uint32_t dst = map_to_cta(smem_u32(smem), (uint32_t)owner) +
                           (uint32_t)(((slot * (W / 4) + (ch * 16 - owner * W) / 4) * 128 + row) * 16);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        st_cluster_v4(dst + (uint32_t)(i * 128 * 16), r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
    }
  }
  cluster_sync_all();
  if (warp >= 2 && ok) {
    const long grow = (long)tm * BM + row;
#pragma unroll
    for (int cc = 0; cc < W / 16; ++cc) {
      const int ch = rank * (W / 16) + cc;
      if ((ch & 1) != half) continue;
      uint32_t r[16];
      tmem_ld_32x32b_x16(taddr + (uint32_t)(ch * 16), r);
      tmem_wait_ld();
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
#pragma unroll
      for (int src = 0; src < S; ++src) {
        if (src == rank) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(r[i]);
        } else {
          const int slot = src < rank ? src : src - 1;
          const float4* from = reinterpret_cast<const float4*>(smem) + (slot * (W / 4) + cc * 4) * 128 + row;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 f = from[i * 128];
            v[4 * i] += f.x; v[4 * i + 1] += f.y; v[4 * i + 2] += f.z; v[4 * i + 3] += f.w;
          }
        }
      }
      if (grow < p.M) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = tn * BN + ch * 16 + h * 8;
          float w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) w[i] = v[h * 8 + i];
          if (col < p.N) finish8(p, grow, col, w);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(acc, C_::TMEM_COLS);
}

// Clusters of S CTAs that the device holds at once (0: none).
template <int BN, int S>
int split_slots() {
  static int slots = -1;
  if (slots >= 0) return slots;
  if (cudaFuncSetAttribute(gemm_bf16_splitk<BN, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)SplitCfg<BN>::SMEM) != cudaSuccess) {
    cudaGetLastError();
    return slots = 0;
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = S;
  cfg.blockDim = kSplitThreads;
  cfg.dynamicSmemBytes = SplitCfg<BN>::SMEM;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_bf16_splitk<BN, S>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  return slots = n;
}

template <int BN, int S>
int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t st) {
  if (split_slots<BN, S>() <= 0) return -4;
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = (unsigned)(tiles * S);
  cfg.blockDim = kSplitThreads;
  cfg.dynamicSmemBytes = SplitCfg<BN>::SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return (int)cudaLaunchKernelEx(&cfg, gemm_bf16_splitk<BN, S>, ta, tb, p);
}
