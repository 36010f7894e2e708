// salsa_space.h -- host side: device memory that a handle keeps, when memory is short.
// The allocator and its release come as arguments, so that this runs without a device.
#pragma once
#include <cstddef>

namespace salsa {

struct Space {
  void *p = nullptr;
  size_t bytes = 0;
};

// Workspaces of the lane form: how many of `grid` blocks (per_block bytes each) it can run
// with; its blocks take their tiles from a counter, so any number works.  The memory that is
// there is kept until more is had.  When memory is short, three quarters or half of the blocks
// do: with fewer the warp form, which needs none (0), is as fast.
template <typename Alloc, typename Release>
int lane_blocks(Space &s, int grid, size_t per_block, Alloc alloc, Release release) {
  if (grid <= 0 || per_block == 0) return 0;
  const int least = (grid + 1) / 2;
  const int tries[3] = {grid, (3 * grid + 3) / 4, least};
  for (int g : tries) {
    if (s.bytes >= (size_t)g * per_block) break;   // as many as that fit already
    if (void *p = alloc((size_t)g * per_block)) {
      if (s.p) release(s.p);
      s.p = p;
      s.bytes = (size_t)g * per_block;
      return g;
    }
  }
  const size_t have = s.bytes / per_block;
  return have >= (size_t)grid ? grid : (have >= (size_t)least ? (int)have : 0);
}

// Cell order lists of n entries: two of them (the second one for moist clear cells), or, when
// memory is short, one, with those cells among the dry ones.  Returns how many, 0 for none.
template <typename Alloc>
int order_lists(size_t n, void **p, Alloc alloc) {
  for (int lists = 2; lists > 0; lists--)
    if ((*p = alloc((size_t)lists * n * sizeof(int)))) return lists;
  return 0;
}

}  // namespace salsa
