// Index rules that kernels share with the CPU tests: plain C++, no CUDA header.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define DG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define DG_HOST_DEVICE inline
#endif

namespace dg {

// Swapped tile family: every how-many-eth k-block of the operand ring the scale warp fetches and publishes scale words (a power of two).
// A word serves new_words k-blocks; on those in between, the weight producer arrives on the stage's barrier in the scale warp's stead.
// Before it arrives, the warp waits until the stage's previous round (k-block n - S of a ring of S stages) is over, and that wait knows
// the parity of the round only: it is right if k-block n - 2 S is known to be over by then.  What is known is what the wait before said,
// that k-block n - period - S is over.  So the period must not exceed S: in a shorter ring the words are fetched anew for every k-block.
// (Waiting for the stages in between as well would be no cure: k-blocks that the warp takes no part in may be over already, a whole
// round ahead, and a wait for the round before would then last for the round after.)  No ring that the rule chooses is that short.
DG_HOST_DEVICE uint32_t scale_period(uint32_t num_stages, uint32_t new_words) { return num_stages < new_words ? 1u : new_words; }

}  // namespace dg
