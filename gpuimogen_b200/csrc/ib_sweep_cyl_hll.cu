// ib_sweep_cyl_hll.cu -- the HLL half of the cylindrical-geometry sweeps (ib_sweep_cyl.cu).
#include "ib_sweep_launch.cuh"

namespace ib {
int launch_sweep_cyl_hll(int slope, double *q, int64_t slab, const int grid[3], SweepStep lambda, double gamma,
                         double rho_min, double c_iso, cudaStream_t st, const CylSweep &cs)
{
    return launch_sweep_cyl_slope<IB_METHOD_HLL>(slope, q, slab, grid, lambda, gamma, rho_min, c_iso, st, cs);
}
}  // namespace ib
