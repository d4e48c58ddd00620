// Shared device-side primitives for the sm_100a kernels of this package:
// mbarrier / TMA / tcgen05 (5th-gen tensor core + tensor memory) PTX wrappers,
// bounded waits with an error word, and small numeric helpers.
//
// Every wait in this file is bounded.  A wait that runs out records a code in
// the library-wide error word (see mmt_error_word) and returns false; callers
// unwind, release tensor memory and return, so the CUDA context stays usable.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define MMT_DEVICE __device__ __forceinline__

// ---------------------------------------------------------------------------
// Error reporting
// ---------------------------------------------------------------------------
// Codes written to the error word by device code (first writer wins).
enum MmtErr : int {
  MMT_OK = 0,
  MMT_ERR_MBAR_TIMEOUT = 1,   // an mbarrier wait ran out
  MMT_ERR_FLAG_TIMEOUT = 2,   // a wait on a flag in (peer) global memory ran out
  MMT_ERR_BOUNDS = 3,         // a debug bounds check failed (access skipped)
  MMT_ERR_TMEM = 4,           // tensor-memory allocation did not come back
};

// One error word per loaded library and device.  Kernels get its device
// address as a parameter (host code resolves it with cudaGetSymbolAddress).
struct MmtErrorWord {
  int code;      // MmtErr
  int where;     // kernel-specific site id
  int block;     // blockIdx.x of the reporter
  int aux;       // extra value (stage, tile, ...)
};

MMT_DEVICE void mmt_report(MmtErrorWord* ew, int code, int where, int aux) {
  if (ew == nullptr) return;
  if (atomicCAS(&ew->code, 0, code) == 0) {
    ew->where = where;
    ew->block = (int)blockIdx.x;
    ew->aux = aux;
    __threadfence_system();
  }
}

MMT_DEVICE uint64_t mmt_globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Default deadline for in-kernel waits (nanoseconds).
#ifndef MMT_WAIT_NS
#define MMT_WAIT_NS 2000000000ull
#endif

// ---------------------------------------------------------------------------
// Programmatic dependent launch (host side: launch_dependent in runtime.h)
// ---------------------------------------------------------------------------
// First statement of a kernel that may be launched while its predecessor in the stream still runs: returns when every
// earlier grid has finished and its writes are visible, then lets the next kernel's CTAs take the SM resources that
// this grid leaves free.  Nothing in front of it may touch global memory (barrier set-up, tensor-memory allocation and
// descriptor prefetches may); EVERY thread block has to execute it, so that "this grid has finished" implies the same
// of all grids before it.
// What such a kernel reads may be written while it already runs, in front of that statement.  So it reads through ordinary
// loads: a pointer parameter that is `const` and `__restrict__` (or __ldg) promises data that does not change during the
// kernel, for which the compiler may use the read-only path, whose lines nothing refreshes, and which it may move up.  The
// same goes for __restrict__ on a buffer that is read and written in place.  Outputs that are only written keep it, which
// is what lets loads pass their stores.
MMT_DEVICE void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
MMT_DEVICE void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
MMT_DEVICE void grid_dependency_sync() {
  grid_dependency_wait();
  grid_dependents_launch();
}

// ---------------------------------------------------------------------------
// Shared-memory address helpers
// ---------------------------------------------------------------------------
MMT_DEVICE uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

MMT_DEVICE uint32_t elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t"
      ".reg .b32 rx;\n\t"
      ".reg .pred px;\n\t"
      "elect.sync rx|px, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, px;\n\t"
      "}\n"
      : "=r"(pred));
  return pred;
}

// ---------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------
MMT_DEVICE void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

MMT_DEVICE void mbar_fence_init() {
  // Make barrier initialisation visible to the async proxy (TMA, tcgen05.commit).
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

MMT_DEVICE void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

MMT_DEVICE void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait on an mbarrier phase.  Returns false after MMT_WAIT_NS and
// records (code, where) in the error word.
MMT_DEVICE bool mbar_wait(uint64_t* bar, uint32_t parity, MmtErrorWord* ew, int where) {
  const uint32_t addr = smem_u32(bar);
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 0x3ff) == 0x3ff) {
      uint64_t now = mmt_globaltimer();
      if (t0 == 0) t0 = now;
      else if (now - t0 > MMT_WAIT_NS) {
        mmt_report(ew, MMT_ERR_MBAR_TIMEOUT, where, (int)parity);
        return false;
      }
    }
  }
}

// The same by a whole warp, with one answer.
MMT_DEVICE bool mbar_wait_warp(uint64_t* bar, uint32_t parity, MmtErrorWord* ew, int where) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, ew, where));
}

// Warp-uniform values.  The operands of tcgen05.mma and of TMA copies live in uniform registers.  A loop that only one
// lane runs (`if (lane == 0)`) computes them per thread and moves every word of every descriptor over, one after the
// other; a loop that the whole warp runs on values the compiler knows to be the same in all lanes keeps them there.
// So the issuing warps run their loops together and elect a lane for the instructions alone.
// Measured: 1024 x 1280 x 3840 (128-row tiles, 64-wide k-blocks) 30.5 -> 24.7 us, 4096 x 1280 x 6848 (256-row tiles)
// 65.6 -> 62.3 us; attention forward and backward of 16384 patches 1.75 -> 1.64 and 7.00 -> 6.28 ms.
MMT_DEVICE int warp_uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
MMT_DEVICE uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

// One non-blocking look at an mbarrier phase (true = that phase has completed).
MMT_DEVICE bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// ---------------------------------------------------------------------------
// TMA (cp.async.bulk.tensor): plain per-CTA loads and stores only.
// ---------------------------------------------------------------------------
MMT_DEVICE void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

MMT_DEVICE void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

MMT_DEVICE void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

MMT_DEVICE void tma_store_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}

MMT_DEVICE void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
MMT_DEVICE void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
MMT_DEVICE void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
MMT_DEVICE void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---------------------------------------------------------------------------
// tcgen05: tensor memory + MMA
// ---------------------------------------------------------------------------
// Allocate `cols` (power of two, >= 32) tensor-memory columns; the base address
// is written to *smem_slot.  Must be called by one full warp.
MMT_DEVICE void tmem_alloc(uint32_t* smem_slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
               ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
}
MMT_DEVICE void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
MMT_DEVICE void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

MMT_DEVICE void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
MMT_DEVICE void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
MMT_DEVICE void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
MMT_DEVICE void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The mbarrier gets one arrival when every tcgen05.mma issued so far by this
// thread has finished reading its operands and writing its accumulator.
MMT_DEVICE void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               ::"r"(smem_u32(bar)) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]; bf16 inputs, fp32 accumulate.
MMT_DEVICE void tc_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]
MMT_DEVICE void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Instruction descriptor for kind::f16 with bf16 A/B and fp32 D.
//   bits [4,6) D format (1 = f32); [7,10) A format (1 = bf16); [10,13) B format;
//   bit 15 A major (0 = K, 1 = MN); bit 16 B major; [17,23) N>>3; [24,29) M>>4.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory matrix descriptor (128-byte swizzle, Blackwell version field 1).
//   bits [0,14) start address >> 4; [16,30) leading byte offset >> 4;
//   [32,46) stride byte offset >> 4; [46,48) version = 1; [61,64) layout (2 = SW128).
// K-major tile [rows][64 bf16]: rows 128 B apart, 8-row groups SBO = 1024 B apart, LBO unused (1).
// MN-major tile [k rows][64 bf16 of MN]: k rows 128 B apart, 8-k-row groups SBO = 1024 B apart,
//   next 64-element MN chunk LBO bytes further.
MMT_DEVICE uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffff) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// The same descriptor split into its 32-bit halves.  Only the low half depends on the tile's address, and moving
// the start address by `bytes` (a multiple of 16) adds bytes >> 4 to it: an MMA issue loop builds both halves
// once and then spends one integer add per instruction instead of re-encoding the descriptor, which matters
// because a single thread has to issue an MMA every ~128 cycles.
MMT_DEVICE uint32_t smem_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3ffff) >> 4) | (((lbo_bytes >> 4) & 0x3fff) << 16);
}
MMT_DEVICE uint32_t smem_desc_hi(uint32_t sbo_bytes) {
  return ((sbo_bytes >> 4) & 0x3fff) | (1u << 14) | (2u << 29);
}
MMT_DEVICE uint64_t smem_desc_join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp gets lane
// (warp%4)*32+i, registers r[0..31] = columns c..c+31.
MMT_DEVICE void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

MMT_DEVICE void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

MMT_DEVICE void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
MMT_DEVICE void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

MMT_DEVICE void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// ---------------------------------------------------------------------------
// Flags in (peer) global memory: release store / bounded acquire spin.
// ---------------------------------------------------------------------------
MMT_DEVICE void flag_store_release_sys(int* flag, int value) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}
MMT_DEVICE int flag_load_acquire_sys(const int* flag) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
  return v;
}
MMT_DEVICE void flag_add_release_sys(int* flag, int value) {
  asm volatile("red.release.sys.global.add.s32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}
// Spin until *flag >= target; false (and an error record) after `limit_ns`.
MMT_DEVICE bool flag_wait_ge(const int* flag, int target, uint64_t limit_ns, MmtErrorWord* ew, int where) {
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    if (flag_load_acquire_sys(flag) >= target) return true;
    if ((it & 0x3f) == 0x3f) {
      uint64_t now = mmt_globaltimer();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) {
        mmt_report(ew, MMT_ERR_FLAG_TIMEOUT, where, target);
        return false;
      }
      __nanosleep(64);
    }
  }
}

// ---------------------------------------------------------------------------
// Numeric helpers
// ---------------------------------------------------------------------------
MMT_DEVICE uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
MMT_DEVICE float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
MMT_DEVICE float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
MMT_DEVICE float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
MMT_DEVICE float gelu_erf(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
MMT_DEVICE float gelu_erf_grad(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.3989422804014327f * __expf(-0.5f * x * x);
  return cdf + x * pdf;
}
MMT_DEVICE float silu(float x) { return x / (1.0f + __expf(-x)); }
