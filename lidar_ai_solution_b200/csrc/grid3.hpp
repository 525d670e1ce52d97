// Extent of a (batched) voxel grid.
#pragma once
#include <stdint.h>

namespace spconvb {

struct Grid3 {
  int32_t g[3];
  int32_t batch;
};

}  // namespace spconvb
