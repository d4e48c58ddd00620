// The loop of one softmax warp of the attention backward kernels over its CTA's score blocks.
//
// The warps of a tensor-memory lane quadrant write P and dS over columns that the others still have to read, so they meet
// at a barrier in every block.  That barrier has no limit, unlike the wait for a block's products in front of it, and the
// clocks of the warps are their own: of four warps that wait for the same products one may run out of time while the others
// see them arrive.  So a warp never leaves the loop early.  Once a wait has run out it does no more work, and comes to the
// barrier of every remaining block all the same; the others, whose products then stop coming, run out in turn.
// (No CUDA in here: the CPU tests compile it with threads in the place of warps.)
#pragma once

#ifdef __CUDACC__
#define MMT_LOOP_FN __device__ __forceinline__
#else
#define MMT_LOOP_FN inline
#endif

namespace attn {

// Per block: wait(block) says whether its products have arrived, work(block) does the block and comes to the barrier once,
// barrier() does nothing else.  False when a wait ran out.
template <class Wait, class Work, class Barrier>
MMT_LOOP_FN bool for_blocks_in_step(int n, const Wait& wait, const Work& work, const Barrier& barrier) {
  bool ok = true;
  for (int it = 0; it < n; ++it) {
    ok = ok && wait(it);
    if (!ok) {
      barrier();
      continue;
    }
    work(it);
  }
  return ok;
}

}  // namespace attn
