// stage_fp32_x.cu -- stage kernels of 1D grids, float instantiation (see stage.cuh, stage1d.cuh).
#include "stage_launch.cuh"

namespace grhd {
template cudaError_t stage_setup_sd<0, float, float>(int, int);
template void launch_stage_sd<0, float, float>(int, int, int, const GridDev *, const BlockMap *, int, cudaStream_t);
template cudaError_t stage1d_setup<float, float>(int, int);
template void launch_stage1d<float, float>(int, int, int, int, const GridDev *, const BlockMap *, int, cudaStream_t);
}  // namespace grhd
