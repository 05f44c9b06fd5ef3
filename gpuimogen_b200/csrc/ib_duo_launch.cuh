// ib_duo_launch.cuh -- host launch logic of the two-cells-a-thread sweep kernels (ib_duo.cuh).
#pragma once

#include "ib_duo.cuh"
#include "ib_internal.cuh"

namespace ib {

template <int METHOD, int SLOPE, typename FT, int TT, int NS, bool ODD, bool FILL, int GEO>
int launch_duo_row_t(const SweepArgs &a, const FluidConsts<FT> &c, cudaStream_t st)
{
    auto kern = duo_row_kernel<METHOD, SLOPE, FT, TT, NS, ODD, FILL, GEO>;
    constexpr size_t shm = duo_smem_bytes<FT, TT>();
    static SmemOptIn record;
    const int rc = opt_in(record, kern, shm);
    if (rc) return rc;
    const int T = (a.nx + 1) / 2, rp = TT / T;
    const int64_t rows = (int64_t)a.ny * a.nz;
    const int64_t nblk = (rows + rp - 1) / rp;
    const int vec = !ODD && !((uintptr_t)a.q & 15) && !(a.slab & 1);
    kern<<<(unsigned)nblk, (rp * T + 31) / 32 * 32, shm, st>>>(a, c, rp, T, vec);
    return check_launch();
}

// x rows of up to 1024 cells.  The thread count is the one that leaves few lanes idle: rows of up to 128
// cells share a CTA of 128 threads, two rows of 129-160 cells one of 160, longer rows have a CTA of their
// own.  Against one thread per cell (HLLC FP64, x of 160^3 / 256^3 / 320 x 100 x 64 / 512 x 512 x 64 / 1000 x
// 100 x 64): 0.142 / 0.535 / 0.078 / 0.607 / 0.312 -> 0.137 / 0.469 / 0.067 / 0.548 / 0.282 ms.
template <int METHOD, int SLOPE, typename FT, int GEO = CYL_NONE>
int launch_duo_row(double *q, int64_t slab, const int grid[3], SweepStep lambda, const FluidConsts<FT> &c,
                   cudaStream_t st, int nsweep, double crin = 0.0, double cdr = 0.0)
{
    const int nx = grid[0];
    if (nx > 1024 || (int64_t)grid[1] * grid[2] >= (int64_t)1 << 31) return IB_ERROR_NOIMPLEMENT;
    const bool fill = lambda.filled && lambda.bc.depth > 0 && nsweep == 1;
    SweepArgs a{q, slab, grid[0], grid[1], grid[2], lambda, crin, cdr, fill ? lambda.bc : RowBc{0, 0, 0}};
    if (fill) *lambda.filled = true;
    const int T = (nx + 1) / 2;
    auto go = [&](auto ns, auto odd, auto fl) {
        auto t = [&](auto tt) {
            return launch_duo_row_t<METHOD, SLOPE, FT, decltype(tt)::value, decltype(ns)::value, decltype(odd)::value,
                                    decltype(fl)::value, GEO>(a, c, st);
        };
        using std::integral_constant;
        if (T <= 64 || (T > 80 && T <= 128)) return t(integral_constant<int, 128>{});
        if (T <= 160) return t(integral_constant<int, 160>{});
        if (T <= 192) return t(integral_constant<int, 192>{});
        if (T <= 256) return t(integral_constant<int, 256>{});
        return t(integral_constant<int, 512>{});
    };
    std::integral_constant<int, 1> one;
    if constexpr (GEO == CYL_NONE) {
        if (nsweep == 2 && !(nx & 1)) return go(std::integral_constant<int, 2>{}, std::false_type{}, std::false_type{});
    }
    if (fill) return (nx & 1) ? go(one, std::true_type{}, std::true_type{}) : go(one, std::false_type{}, std::true_type{});
    for (int k = 0; k < nsweep; k++) {
        const int rc = (nx & 1) ? go(one, std::true_type{}, std::false_type{}) : go(one, std::false_type{}, std::false_type{});
        if (rc) return rc;
    }
    return IB_SUCCESSFUL;
}

template <int METHOD, int SLOPE, typename FT, int DIR, int TT, int COLS, bool ODD, int GEO>
int launch_duo_pencil_t(const SweepArgs &a, const FluidConsts<FT> &c, int n, cudaStream_t st, const CylPencil &cyl)
{
    auto kern = duo_pencil_kernel<METHOD, SLOPE, FT, DIR, TT, COLS, ODD, GEO>;
    constexpr size_t shm = duo_smem_bytes<FT, TT>();
    static SmemOptIn record;
    const int rc = opt_in(record, kern, shm);
    if (rc) return rc;
    const int64_t np = (int64_t)a.nx * a.ny * a.nz / n;
    kern<<<(unsigned)((np + COLS - 1) / COLS), ((n + 1) / 2 * COLS + 31) / 32 * 32, shm, st>>>(a, c, np, cyl);
    return check_launch();
}

// y and z pencils, any nx and alignment: as many neighbouring pencils as 256 threads hold, at most 8.  FP64 up to
// 512 cells, the FP32 flux up to 256: above, one pencil's CTA reads 8 bytes of every 32-byte sector, which the FP32
// flux waits for, and four pencils a CTA in the tile kernel are the faster form (us, tile / here: 63 x 257 x 259 y
// 214 / 251, 64 x 403 x 162 y 210 / 295, 601 x 18 x 384 z 209 / 254, 63 x 130 x 512 z 209 / 243; FP64 there 317 / 314,
// 277 / 337, 319 / 315, 316 / 285).
template <int METHOD, int SLOPE, typename FT, int DIR, int GEO = CYL_NONE>
int launch_duo_pencil(double *q, int64_t slab, const int grid[3], SweepStep lambda, const FluidConsts<FT> &c,
                      cudaStream_t st, int nsweep, CylPencil cyl = CylPencil{0.0, 0.0, 0, 0})
{
    const int n = grid[DIR - 1];
    if (n > (sizeof(FT) == 4 ? 256 : 512) || (int64_t)grid[0] * grid[1] * grid[2] / n >= (int64_t)1 << 31)
        return IB_ERROR_NOIMPLEMENT;
    SweepArgs a{q, slab, grid[0], grid[1], grid[2], lambda, 0.0, 0.0, RowBc{0, 0, 0}};
    using std::integral_constant;
    auto go = [&](auto odd) {
        auto t = [&](auto tt, auto cols) {
            return launch_duo_pencil_t<METHOD, SLOPE, FT, DIR, decltype(tt)::value, decltype(cols)::value,
                                       decltype(odd)::value, GEO>(a, c, n, st, cyl);
        };
        if (n > 256) return t(integral_constant<int, 256>{}, integral_constant<int, 1>{});
        if (n > 128) return t(integral_constant<int, 256>{}, integral_constant<int, 2>{});
        if (n > 64) return t(integral_constant<int, 256>{}, integral_constant<int, 4>{});
        if (n > 32) return t(integral_constant<int, 256>{}, integral_constant<int, 8>{});
        return t(integral_constant<int, 128>{}, integral_constant<int, 8>{});
    };
    for (int k = 0; k < nsweep; k++) {
        const int rc = (n & 1) ? go(std::true_type{}) : go(std::false_type{});
        if (rc) return rc;
    }
    return IB_SUCCESSFUL;
}

}  // namespace ib
