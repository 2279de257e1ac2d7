// The work of a CTA that goes through several items of a launch one after another.
//
// The tensor-core kernels fit one CTA per SM, so nothing else runs there while a CTA sets up, fills
// its pipeline, drains it and writes its rows: 3 us, against 1 us per K/V tile of work. A CTA
// that takes several items keeps its copies and products running across them.
//
// The items come longest first; CTA c takes one from each run of gridDim.x, alternately from the
// run's front and its back, which gives every CTA nearly the same number of tiles (within 1 % of
// what longest-first dispatch by the hardware gives, for 3000 to 32768 causal rows of 32 heads). In
// time that holds for short walks only: in long ones the CTAs drift apart (see dq_loops). The
// threads of a CTA decode its items side by side into shared memory at the start; the warps read
// them from there.
#pragma once
#include <stdint.h>

namespace spa {

struct alignas(16) WorkItem {
  int h, b;   // head, batch
  int r0;     // first row of the stationary tile in its sequence
  int sg;     // sequence of a packed batch
  int n0;     // tiles of the streamed operand
};

__device__ __forceinline__ int item_index(int pos) {
  return pos * gridDim.x + ((pos & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}
// Items of this CTA.
__device__ __forceinline__ int item_count(int n_items) {
  const int full = n_items / gridDim.x;
  return full + (item_index(full) < n_items ? 1 : 0);
}

// Host: CTAs for a launch of n_items, at most max_items each.
inline long long worklist_grid(long long n_items, int n_sm, int max_items) {
  if (n_items <= n_sm) return n_items;
  const long long rounds = (n_items + (long long)n_sm * max_items - 1) / ((long long)n_sm * max_items);
  return n_sm * rounds;
}

}  // namespace spa
