// cell_launch.cuh -- host launcher of the stage cell kernel, instantiated per precision in
// cell_fp64.cu / cell_fp32.cu (each precision compiled with its own floating-point flags,
// the same as the face kernels and the persistent kernel of that precision).
#pragma once

#include "flux_launch.h"
#include "cell.cuh"

namespace grhd {

static_assert(CELL_BS == 1 << CELL_LB && CELL_BS_WIDE == 1 << CELL_LB_WIDE, "block sizes are the kernel's");

template <int LB, class R, class PT>
inline void launch_cell_lb(int mode, const GridDev *grids, const BlockMap *map, unsigned nb, int dirs, cudaStream_t s) {
  constexpr int bs = 1 << LB;
  const size_t smem = cell_smem_bytes<R, PT, LB>(dirs);
  switch (mode) {
    case 0: k_cell_update<0, R, PT, LB><<<nb, bs, smem, s>>>(grids, map); break;
    case 1: k_cell_update<1, R, PT, LB><<<nb, bs, smem, s>>>(grids, map); break;
    case 2: k_cell_update<2, R, PT, LB><<<nb, bs, smem, s>>>(grids, map); break;
    default: k_cell_update<3, R, PT, LB><<<nb, bs, smem, s>>>(grids, map); break;
  }
}
// dirs: the most active directions of any grid in the launch (sizes the staging buffers);
// wide: 256-thread blocks (FP64 only)
template <class R, class PT>
void launch_cell(int mode, bool wide, const GridDev *grids, const BlockMap *map, int nblocks, int dirs, cudaStream_t s) {
  if (nblocks <= 0) return;
  if constexpr (sizeof(PT) == sizeof(double)) {
    if (wide) {
      launch_cell_lb<CELL_LB_WIDE, R, PT>(mode, grids, map, (unsigned)nblocks, dirs, s);
      return;
    }
  }
  launch_cell_lb<CELL_LB, R, PT>(mode, grids, map, (unsigned)nblocks, dirs, s);
}

}  // namespace grhd
