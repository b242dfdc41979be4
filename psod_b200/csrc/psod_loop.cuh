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

// The queue of ready blocks is a ring of as many places as blocks were active
// at the launch, which may be a handful, so that places are reused while
// consumers of the lap before are still at them.  A value is put into an empty
// place and taken out by an exchange: whichever consumer of a place exchanges
// first has the value, no other one sees it, and each of them gets one, as many
// values being put into a place as consumers were sent to it.  (Read first and
// emptied afterwards, a value could be seen by the consumer a lap later too.)
// Mem: load, exchange and compare-and-swap of a word shared by the CTAs.
constexpr unsigned RING_EMPTY = 0xffffffffu;

template <class Mem>
PSOD_LOOP_FN bool ring_put(Mem &m, unsigned *place, unsigned block) {
  return m.cas(place, RING_EMPTY, block) == RING_EMPTY;
}

template <class Mem>
PSOD_LOOP_FN bool ring_take(Mem &m, unsigned *place, unsigned &block) {
  if (m.load(place) == RING_EMPTY) return false;
  block = m.exchange(place, RING_EMPTY);
  return block != RING_EMPTY;
}

// Place e of a box of sx by sy by any planes, total places in all, as (x, y, z).
// Below 2^22 places the quotient through FP32 is exact: e + 1/2 is, the rounded
// reciprocal and product are off by less than e / s * 2^-23 < 1 / (2 s), and the
// quotient lies at least that far from a whole number.  Larger boxes divide
// (blocks of one cell and ncut from 21: windows up to (4 ncut + 1)^3 places).
PSOD_LOOP_FN void box_split(int e, int sx, int sy, int total, int &x, int &y, int &z) {
  int q;
  if (total <= (1 << 22)) {
    q = (int)(((float)e + 0.5f) * (1.0f / (float)sx));
    z = (int)(((float)q + 0.5f) * (1.0f / (float)sy));
  } else {
    q = e / sx;
    z = q / sy;
  }
  x = e - q * sx;
  y = q - z * sy;
}

}  // namespace psod
