// How many CTAs the resident CG of a small system takes (plain C++, no CUDA).
#pragma once

#include <stdint.h>

#include <initializer_list>

namespace ufc {

constexpr int64_t kOneCtaSlices = 4;    // up to here one CTA
constexpr int64_t kClusterSlices = 48;  // up to here one cluster
constexpr int kResCluster = 16;         // CTAs of a cluster at most (a non-portable size)
constexpr int kResPortable = 8;         // the largest size that every device of the architecture takes

// CTAs for a system of `slices` slices, or 0 for the chain of kernels.
// placeable(ctas) says whether the device can hold a cluster of that many now: a
// GPU with few SMs in a GPC (partitioned, or shared with others) need not take
// 16 of them.  8 CTAs then own up to 6 slices each, within the 16 of a CTA.
template <class Placeable>
inline int resident_ctas(int64_t slices, Placeable placeable) {
  if (slices <= kOneCtaSlices) return 1;
  if (slices > kClusterSlices) return 0;
  for (int most : {kResCluster, kResPortable}) {
    const int g = (int)(slices < most ? slices : most);
    if (placeable(g)) return g;
  }
  return 0;
}

}  // namespace ufc
