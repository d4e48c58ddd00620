// Host-side runtime shared by every translation unit of the kernel library.
#pragma once
#include <cuda_runtime.h>

struct MmtErrorWord;

// Number of SMs of the current device (cached).
int mmt_sm_count();
// Device address of the library's error word for the current device
// (allocated on first use; kernels record bounded-wait failures there).
MmtErrorWord* mmt_error_word();

// Makes sure the calling thread has the CUDA context of the device that owns `ptr` (first call per thread).
int mmt_ensure_context(const void* ptr);

// Launches a kernel that starts with grid_dependency_sync() (common.cuh) so that its CTAs may become resident while the
// previous kernel of the stream drains: the launch latency, the prologue and the previous grid's tail overlap instead
// of following one another.  A training step is up to 1400 launches with about a microsecond between two of them.
// Measured: 896 x 896 vision step (1105 launches) 30.95 -> 29.24 ms, 32-layer encoder without gradients on 256 patches
// 6.31 -> 6.20 ms; no difference where the kernels are long (text step of 2048 tokens 17.28 and 17.27 ms).
template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// One sum of partial rows: out[c] (+)= sum over parts of partial[part][c] (fp32 -> bf16).
struct MmtReduceSegment {
  const float* partial;
  void* out;
  int parts, cols, accumulate;
};
#define MMT_MAX_REDUCE_SEGMENTS 6

extern "C" {
// Copies the error word to out[4] = {code, where, block, aux}; synchronises the device.
int mmt_get_error(int* out);
// Device address of the error word ([4] int32), or nullptr if it could not be allocated.
void* mmt_error_word_address();
// Resets the error word to zero.
int mmt_clear_error();
// Library build tag, for tests that check the native path is loaded.
const char* mmt_version();
}
