// The X ring of the tcgen05 kernels on the way out after an abort: which copies into this CTA's shared memory may still be in
// flight, and what their barriers need to complete.  Plain C++, so that it can be tested without a GPU.
//
// NPW producer warps bring the items (batch tiles) 0, 1, 2, ... into NXS stages, item j into stage j % NXS.  NSH consecutive warps share an
// item: the warps p with p / NSH == j % (NPW / NSH).  Each of them announces its own bytes with one arrival at the stage's barrier,
// which expects NSH.  A warp announces an item only when the stage's previous item has been consumed, and stops for good at the first one for
// which the abort flag is up.
#pragma once

#ifdef __CUDACC__
#define HASTE_RING_HD __host__ __device__
#else
#define HASTE_RING_HD
#endif

namespace haste {

// The item whose bytes a stage may still be waiting for: the latest that any warp announced (-1: none ever), and how many of
// the warps that share it did not.  With that many arrivals in their place the barrier's phase ends when the announced bytes have landed.  (The
// phases before it are over: the item before was consumed.)
struct RingDrain { int item, missing; };

template <int NXS, int NPW, int NSH, class LastItem>      // last(p): the last item warp p announced, -1 if none
HASTE_RING_HD inline RingDrain ring_drain(int stage, LastItem last) {
  constexpr int STEP = NPW / NSH;
  RingDrain d = {-1, 0};
  for (int p = 0; p < NPW; ++p) {
    // a warp's items are STEP apart; of any NXS of them in a row one lies in the stage, if any does
    int j = last(p);
    for (int n = 0; n < NXS && j >= 0 && j % NXS != stage; ++n) j -= STEP;
    if (j >= 0 && j % NXS == stage && j > d.item) d.item = j;
  }
  if (d.item >= 0)
    for (int p = d.item % STEP * NSH; p < (d.item % STEP + 1) * NSH; ++p) d.missing += last(p) < d.item;
  return d;
}

}  // namespace haste
