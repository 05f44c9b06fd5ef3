// ib_sweep_cyl.cu -- the cylindrical-geometry sweeps (HLLC here, HLL in ib_sweep_cyl_hll.cu, FP64) with the
// geometry's update (ib_cyl.cuh): radial x sweeps in the two-cell row kernel (rows up to 1024 cells),
// theta y sweeps in the pencil-pair kernel (pencils up to 256 cells, x even) or the two-cell pencil
// kernel (up to 512), the tile kernel for longer ones.
#include "ib_sweep_launch.cuh"

namespace ib {
int launch_sweep_cyl_hll(int slope, double *q, int64_t slab, const int grid[3], SweepStep lambda, double gamma,
                         double rho_min, double c_iso, cudaStream_t st, const CylSweep &cs);

int launch_sweep_cyl(int method, int slope, double *q, int64_t slab, const int grid[3], SweepStep lambda,
                     double gamma, double rho_min, double c_iso, cudaStream_t st, const CylSweep &cs)
{
    if (method == IB_METHOD_HLLC)
        return launch_sweep_cyl_slope<IB_METHOD_HLLC>(slope, q, slab, grid, lambda, gamma, rho_min, c_iso, st, cs);
    if (method == IB_METHOD_HLL)
        return launch_sweep_cyl_hll(slope, q, slab, grid, lambda, gamma, rho_min, c_iso, st, cs);
    return IB_ERROR_INVALID_ARGS;
}
}  // namespace ib
