// region_rows.h -- how many CTAs of a cloud-region launch get rows in global
// memory.  The kernels stride over their columns, so any number of CTAs from
// one up computes the same values.
#pragma once

#include <algorithm>
#include <cstddef>

namespace socgpu {

// The most that the rows of one launch take: what 152 CTAs need for the
// tallest columns (512 layers, infra-red, three regions, FP64: 1485 MB), so
// that no column height costs resident CTAs there; 137 layers need 407 MB at
// most.
constexpr size_t kRegionRows = (size_t)1536 << 20;

// The CTAs, of `ctas` wanted, whose rows of `stride` bytes each stay within
// that: at least one, if any are wanted.
inline long long region_grid(long long ctas, size_t stride) {
  return std::min(ctas, std::max<long long>(1, (long long)(kRegionRows / std::max<size_t>(stride, 1))));
}

// Memory for the rows from alloc(bytes) -> bool; where there is none, for half
// as many CTAs, down to one.  False: not even that.
template <class Alloc>
bool take_rows(long long &grid, size_t stride, Alloc alloc) {
  while (!alloc(stride * (size_t)grid)) {
    if (grid <= 1) return false;
    grid = (grid + 1) / 2;
  }
  return true;
}

}  // namespace socgpu
