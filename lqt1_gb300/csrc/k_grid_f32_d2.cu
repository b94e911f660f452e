// k_grid_f32_d2.cu -- occupancy variants of the 2D mixed-form step kernel
// (separate translation unit so the variants compile in parallel).
#include "k_grid.cuh"

namespace lqt {

cudaError_t launch_f32_d2(const GridDev<float> &gd, const StepT<float> &kk, int cur, int minb, cudaStream_t st)
{
    if (gd.plist) {
        k_grid_step_list<float, 2><<<grid_list_blocks(gd.ntissue), 256, 0, st>>>(gd, kk, cur);
        return cudaGetLastError();
    }
    if (gd.fold) return grid_step_launch<float, 2, 4, 64, true>(gd, kk, cur, st);
    if (minb >= kGridPipe) return grid_step_pipe_launch<2>(gd, kk, cur, st);
    if (minb >= 4) return grid_step_launch<float, 2, 4, 256>(gd, kk, cur, st);
    if (minb == 3) return grid_step_launch<float, 2, 3, 256>(gd, kk, cur, st);
    return grid_step_launch<float, 2, 2, 256>(gd, kk, cur, st);
}

}  // namespace lqt
