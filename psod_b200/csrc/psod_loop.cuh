// psod_loop.cuh -- the words that the CTAs of the device seed loop
// (psod_sod.cu) exchange, as plain functions: the host compiles them too, so
// that their rules are tested without a GPU.
#pragma once

#ifdef __CUDACC__
#define PSOD_LOOP_FN __host__ __device__ __forceinline__
#else
#define PSOD_LOOP_FN inline
#endif

namespace psod {

// A shared refinement is one 64-bit word: its item count above, the next item
// below.  A warp draws with one atomicAdd of 1 and learns both from the value
// that it got, so an accepted item belongs to the refinement that the word
// held at the draw, whatever the owner has published since; a refinement of
// no items (0) is a closed one.  The owner closes it only after every accepted
// item was finished.  Draws past the end only raise the lower half, which the
// next refinement resets: one draw a warp and visit, far from 2^32.
PSOD_LOOP_FN unsigned long long refine_open(unsigned nitem) { return (unsigned long long)nitem << 32; }

PSOD_LOOP_FN bool refine_take(unsigned long long drawn, unsigned &item) {
  item = (unsigned)drawn;
  return item < (unsigned)(drawn >> 32);
}

}  // namespace psod
