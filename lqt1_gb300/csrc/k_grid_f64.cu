// k_grid_f64.cu -- grid kernels for the FP64 form: launchers, occupancy
// variants and the pseudo-ECG.
#include "k_grid.cuh"

namespace lqt {

template <> cudaError_t launch_grid_step_minb<double>(const GridDev<double> &gd, const StepT<double> &kk, int cur,
                                                      int dim, int minb, cudaStream_t st)
{
    if (gd.plist) return cudaErrorInvalidValue;   // the surrogate's voxel list exists in the mixed form only
    // CTAs of 64: the FP64 pipe sets the pace at any occupancy, and the last
    // wave of wide CTAs runs nearly empty (78k voxels in 305 CTAs of 256 on 152
    // SMs: 684 us a step, 666 us in CTAs of 64)
    if (dim == 1) return grid_step_launch<double, 1, 4, 64>(gd, kk, cur, st);
    if (dim == 2)
        return minb >= 2 ? grid_step_launch<double, 2, 8, 64>(gd, kk, cur, st)
                         : grid_step_launch<double, 2, 4, 64>(gd, kk, cur, st);
    return minb >= 2 ? grid_step_launch<double, 3, 8, 64>(gd, kk, cur, st)
                     : grid_step_launch<double, 3, 4, 64>(gd, kk, cur, st);
}

template <> cudaError_t launch_grid_step<double>(const GridDev<double> &gd, const StepK &k, int cur, int dim, int minb,
                                                 cudaStream_t st)
{
    if (gd.ntissue <= 0) return cudaSuccess;
    return launch_grid_step_minb<double>(gd, step_as<double>(k), cur, dim, minb, st);
}

template <> cudaError_t launch_ghost<double>(const GridDev<double> &gd, int cur, int clock, cudaStream_t st)
{
    int64_t nb = (gd.nbnd + 255) / 256;
    if (nb < 1) nb = 1;
    if (nb > 152 * 16) nb = 152 * 16;
    k_ghost<double><<<(unsigned)nb, 256, 0, st>>>(gd, cur, clock);
    return cudaGetLastError();
}

template <>
cudaError_t launch_ecg<double>(const GridDev<double> &gd, int cur, const float4 *el, int nel, double *partial,
                               double *out, double *t_out, int64_t *counter, int64_t cap, int dim, cudaStream_t st)
{
    const int64_t nb = ecg_blocks(gd.ntissue);
    if (dim == 1) k_ecg_partial<double, 1><<<(unsigned)nb, 256, 0, st>>>(gd, gd.vg[cur], el, nel, partial);
    else if (dim == 2) k_ecg_partial<double, 2><<<(unsigned)nb, 256, 0, st>>>(gd, gd.vg[cur], el, nel, partial);
    else k_ecg_partial<double, 3><<<(unsigned)nb, 256, 0, st>>>(gd, gd.vg[cur], el, nel, partial);
    k_ecg_final<<<nel, 256, 0, st>>>(partial, nb, nel, out, t_out, counter, cap, gd.clk + cur);
    return cudaGetLastError();
}

}  // namespace lqt
