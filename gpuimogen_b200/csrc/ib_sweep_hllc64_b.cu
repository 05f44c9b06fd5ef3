// ib_sweep_hllc64_b.cu -- instantiates the fused sweep kernels for method IB_METHOD_HLLC with double flux arithmetic, the
// second half of the limiters.
#include "ib_sweep_launch.cuh"

namespace ib {
int launch_hllc64_b(int slope, int dir, double *q, int64_t slab, const int grid[3], SweepStep lambda, double gamma,
              double rho_min, double c_iso, cudaStream_t st, int nsweep)
{
    return launch_sweep_slope<IB_METHOD_HLLC, double, 1>(slope, dir, q, slab, grid, lambda, gamma, rho_min, c_iso, st, nsweep);
}
}  // namespace ib
