// ib_ensemble.cu -- batched ensemble of independent 1-D problems in one persistent launch.
//
// Each problem is what the reference runs as a one-dimensional fluid: per iteration the CFL
// timestep (cflTimestep.cu:107-252; in 1-D the HLL template, |p_x| only, halved for HLL/HLLC),
// dt = CFL * tau with the last-step clip (TimeManager.m:124-186), then the forward and the
// backward fluid step, each the 1-D shortcut of performFluidUpdate_3D (flux.cu:52-68): one x
// sweep followed by the boundary fill, and t += 2 dt with Kahan compensation
// (TimeManager.m:270-277).  Here a CTA takes a problem from a device work counter and runs it to
// its end without leaving the kernel; the problem's cells stay in L2 between sweeps (one
// problem is at most a few hundred KB), so the launch reads and writes HBM about once per cell.
// The per-cell arithmetic is the library's sweep arithmetic (stage_prims / stage_faces / stage_flux in
// ens_stages, the two-cell stages of ib_duo.cuh in ens_sweep_two), CFL and boundary code.  A problem's bits
// depend neither on the launch shape nor on how many problems share the launch.  In the strict build they are those
// of the problem run alone through the library's 1-D entry points; in the product build, whose other sweeps do not
// round every product, they agree with them to 1e-12 (relative L1).
#include "ib_bc.cuh"
#include "ib_cfl.cuh"
#include "ib_internal.cuh"
#include "ib_duo.cuh"

namespace ib {

struct EnsArgs {
    double *q;
    int64_t S;
    const int64_t *off;
    const double *h;
    const int32_t *order;
    double *t_out;
    int32_t *it_out;
    unsigned int *counter;
    int32_t np;
    int32_t bc0, bc1;
    int32_t itermax;
    int32_t target;    // chunk length to aim for
    int32_t lcap;      // tile rows (chunk + 8 halo cells) the shared memory planes hold, <= threads
    double gg1;        // gamma (gamma - 1), soundspeed
    double cfl, t_end;
    int32_t halve;
};

// Boundary fill of one 1-D problem after a sweep (setFluidBoundary along x), both sides in order.
__device__ __forceinline__ void ens_boundary(double *qb, int64_t S, int n, int bc0, int bc1)
{
    for (int side = 0; side < 2; side++) {
        const int mode = side ? bc1 : bc0;
        if (mode == IB_BC_OUTFLOW) {
            outflow_x(qb, S, 1, n, side, 1, 4);
        } else if (mode == IB_BC_MIRROR || mode == IB_BC_CONST || mode == IB_BC_LINEAR) {
            for (int k = 0; k < 5; k++) sas_x(qb + k * S, 1, n, mode, side, k == 2, 4);
        }
    }
}

// Number of chunks for a problem of n cells: chunk ch covers cells [ch n / nc, (ch + 1) n / nc), so
// no chunk is longer than the target and, as the in-place rules need, none is shorter than 8 cells.
// Every output cell is the same function of the 9 original cells around it whatever the chunks.
__device__ __forceinline__ int ens_nchunks(int n, int target)
{
    int nc = max(1, (n + target - 1) / target);
    while (nc > 1 && n / nc < 8) nc--;
    return nc;
}

// Stores after a chunk's inputs have been read: the previous chunk's last four outputs, this chunk's output m
// (the last four, and the first chunk's first four, wait), and at the end those still waiting.  pend: two
// buffers, so that a chunk's own outputs do not overwrite those of the chunk before.
__device__ __forceinline__ void ens_store_pending(double *qb, int64_t S, int ch, int cb, int i, const double *pend)
{
    if (ch == 0 || i >= 4) return;
    const double *p = pend + 20 * ((ch - 1) & 1);
#pragma unroll
    for (int k = 0; k < 5; k++) qb[(int64_t)k * S + cb - 4 + i] = p[k * 4 + i];
}
__device__ __forceinline__ void ens_store(double *qb, int64_t S, int ch, int cb, int len, bool single, int m,
                                          const double (&out)[5], double *pend, double *first)
{
    if (!single && ch == 0 && m < 4) {
#pragma unroll
        for (int k = 0; k < 5; k++) first[k * 4 + m] = out[k];
    } else if (!single && m >= len - 4) {
        double *p = pend + 20 * (ch & 1);
#pragma unroll
        for (int k = 0; k < 5; k++) p[k * 4 + m - (len - 4)] = out[k];
    } else {
#pragma unroll
        for (int k = 0; k < 5; k++) qb[(int64_t)k * S + cb + m] = out[k];
    }
}
__device__ __forceinline__ void ens_store_ends(double *qb, int64_t S, int n, int nchunks, int i, const double *pend,
                                               const double *first)
{
    __syncthreads();
    if (nchunks > 1 && i < 4) {
        const double *p = pend + 20 * ((nchunks - 1) & 1);
#pragma unroll
        for (int k = 0; k < 5; k++) {
            qb[(int64_t)k * S + n - 4 + i] = p[k * 4 + i];
            qb[(int64_t)k * S + i] = first[k * 4 + i];
        }
    }
    __syncthreads();
}

// Products that leave a cell are rounded (RN), here and in the form with two rows a thread, and this file is compiled
// without contraction of the rest: otherwise the compiler takes some of them into the sums of the thread that
// formed them, and a cell's result would depend on the form.
//
// Both stages of one chunk, row i of its tr rows a thread, which keeps that cell's state u in registers: on
// return u is the output of rows 4 .. tr - 5.  Two shared-memory planes of FT swap roles between the stages.
template <int METHOD, int SLOPE, typename FT, typename OPS>
__device__ __forceinline__ bool ens_stages(double (&u)[5], int i, int tr, double lambda, const FluidConsts<FT> &c, FT *SA, FT *SB,
                                           int TR)
{
    double u1[5];
    V5<FT> keep;
    bool suspect = false;
    // ---- stage A: prims and fluxes in SA, left faces in SB ----
    if (i < tr) {
        V5<FT> w = stage_prims<METHOD, 1, FT, true, OPS>(u, c);  // HLL floors u
        if constexpr (kPoison<OPS, FT>) suspect = cell_suspect(u[0], w.a[3]);
#pragma unroll
        for (int k = 0; k < 5; k++) SA[k * TR + i] = w.a[k];
    }
    __syncthreads();
    if (i >= 1 && i <= tr - 2) {
        V5<FT> w, dl, dr, L;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            w.a[k] = SA[k * TR + i];
            dl.a[k] = w.a[k] - SA[k * TR + i - 1];
            dr.a[k] = SA[k * TR + i + 1] - w.a[k];
        }
        stage_faces<METHOD, SLOPE, FT, OPS, true>(c, w, dl, dr, L, keep);
#pragma unroll
        for (int k = 0; k < 5; k++) SB[k * TR + i] = L.a[k];
    }
    __syncthreads();
    if (i >= 1 && i <= tr - 3) {
        V5<FT> Lr;
#pragma unroll
        for (int k = 0; k < 5; k++) Lr.a[k] = SB[k * TR + i + 1];
        keep = stage_flux<METHOD, FT, true, OPS>(c, keep, Lr);
#pragma unroll
        for (int k = 0; k < 5; k++) SA[k * TR + i] = keep.a[k];
    }
    __syncthreads();
    if (i >= 2 && i <= tr - 3) {
#pragma unroll
        for (int k = 0; k < 5; k++) u1[k] = sub_product(u[k], lambda, (double)keep.a[k] - (double)SA[k * TR + i - 1]);
    }
    // ---- stage B: prims and fluxes in SB, left faces in SA (no barrier: stage A's last
    // phase read SA only) ----
    if (i >= 2 && i <= tr - 3) {
        V5<FT> w = stage_prims<METHOD, 1, FT, true, OPS>(u1, c);  // HLL floors u1
        if constexpr (kPoison<OPS, FT>) suspect = suspect || cell_suspect(u1[0], w.a[3]);
#pragma unroll
        for (int k = 0; k < 5; k++) {
            SB[k * TR + i] = w.a[k];
            u[k] = u1[k] + u[k];  // the output's (u1 + u0), rounded as it is there first
        }
    }
    __syncthreads();
    if (i >= 3 && i <= tr - 4) {
        V5<FT> w, dl, dr, L;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            w.a[k] = SB[k * TR + i];
            dl.a[k] = w.a[k] - SB[k * TR + i - 1];
            dr.a[k] = SB[k * TR + i + 1] - w.a[k];
        }
        stage_faces<METHOD, SLOPE, FT, OPS, true>(c, w, dl, dr, L, keep);
#pragma unroll
        for (int k = 0; k < 5; k++) SA[k * TR + i] = L.a[k];
    }
    __syncthreads();
    if (i >= 3 && i <= tr - 5) {
        V5<FT> Lr;
#pragma unroll
        for (int k = 0; k < 5; k++) Lr.a[k] = SA[k * TR + i + 1];
        keep = stage_flux<METHOD, FT, true, OPS>(c, keep, Lr);
#pragma unroll
        for (int k = 0; k < 5; k++) SB[k * TR + i] = keep.a[k];
        if constexpr (kPoison<OPS, FT>) suspect = suspect || keep.a[0] != keep.a[0];
    }
    if constexpr (kPoison<OPS, FT>) suspect = __syncthreads_or(suspect);
    else __syncthreads();
    if (i >= 4 && i <= tr - 5) {
#pragma unroll
        for (int k = 0; k < 5; k++) u[k] = .5 * sub_product(u[k], lambda, (double)keep.a[k] - (double)SB[k * TR + i - 1]);
    }
    return suspect;
}

// The same with the IEEE operations, out of line: its registers are not the caller's
template <int METHOD, int SLOPE, typename FT>
__device__ __noinline__ void ens_stages_ieee(double (&u)[5], int i, int tr, double lambda, FluidConsts<FT> c, FT *SA, FT *SB,
                                             int TR)
{
    ens_stages<METHOD, SLOPE, FT, IeeeOps>(u, i, tr, lambda, c, SA, SB, TR);
}

// One x sweep of a problem of n cells in nc chunks (ens_nchunks; the longest chunk + 8 <= lcap <= NT):
// the tile sweep's in-place rules (each chunk loads its cells and 4 halo cells a side of the original
// state; the last four outputs of a chunk wait in `pend` until the next chunk has been computed, the
// first chunk's first four in `first` until the last chunk has read them through the periodic
// wrap).  A chunk's inputs stay in memory until its operands have been tested, so that it can be computed again with the
// IEEE operations.  The arithmetic is the library's sweep arithmetic (stage_prims /
// stage_faces / stage_flux), so the results are those of the tile sweep.
template <int METHOD, int SLOPE, typename FT, int NT>
__device__ __forceinline__ void ens_sweep(double *qb, int64_t S, int n, int nchunks, double lambda,
                                          const FluidConsts<FT> &c, FT *SA, FT *SB, int TR, double *pend,
                                          double *first)
{
    const int i = threadIdx.x;
    const bool single = (nchunks == 1);
    for (int ch = 0; ch < nchunks; ch++) {
        const int cb = (int)((int64_t)ch * n / nchunks);
        const int len = (int)((int64_t)(ch + 1) * n / nchunks) - cb;
        const int tr = len + 8;
        auto fetch = [&](double (&u)[5]) {
            if (i < tr) {
                const int cell = mod_n(cb - 4 + i, n);
#pragma unroll
                for (int k = 0; k < 5; k++) u[k] = qb[(int64_t)k * S + cell];
            }
        };
        double out[5];
        fetch(out);
        __syncthreads();  // every thread is done with the planes
        if (ens_stages<METHOD, SLOPE, FT, FastOps>(out, i, tr, lambda, c, SA, SB, TR)) {
            double x[5];
            fetch(x);
            __syncthreads();
            ens_stages_ieee<METHOD, SLOPE, FT>(x, i, tr, lambda, c, SA, SB, TR);
#pragma unroll
            for (int k = 0; k < 5; k++) out[k] = x[k];
        }
        const bool mine = i >= 4 && i <= tr - 5;
        // every thread has read this chunk's inputs
        ens_store_pending(qb, S, ch, cb, i, pend);
        if (mine) ens_store(qb, S, ch, cb, len, single, i - 4, out, pend, first);
    }
    ens_store_ends(qb, S, n, nchunks, i, pend, first);
}

// The same sweep with two rows a thread: thread t computes rows 2t and 2t + 1 of a chunk (ib_duo.cuh; the edge
// rows' results are not used), TT threads for chunks of up to 2 TT - 8 cells.  Products are rounded (RN), so that
// a cell's result does not depend on which of the two rows it is, and with it not on the chunk length.
template <int METHOD, int SLOPE, typename FT, int TT>
__device__ __forceinline__ void ens_sweep_two(double *qb, int64_t S, int n, int nchunks, double lambda,
                                          const FluidConsts<FT> &c, FT *planes, double *SS, double *pend, double *first)
{
    const int t = threadIdx.x;
    const bool single = (nchunks == 1);
    DuoPos p;
    p.own = t;
    p.left = (t > 0) ? t - 1 : t;
    p.right = (t < TT - 1) ? t + 1 : t;
    p.first = p.ghost = false;
    for (int ch = 0; ch < nchunks; ch++) {
        const int cb = (int)((int64_t)ch * n / nchunks);
        const int len = (int)((int64_t)(ch + 1) * n / nchunks) - cb;
        const int tr = len + 8;
        auto fetch = [&](int i, double (&u)[5]) {
            const int cell = mod_n(cb - 4 + i, n);
#pragma unroll
            for (int k = 0; k < 5; k++) u[k] = (i < tr) ? qb[(int64_t)k * S + cell] : 1.0;
        };
        double ua[5], ub[5];
        fetch(2 * t, ua);
        fetch(2 * t + 1, ub);
        __syncthreads();  // every thread is done with the planes
        const auto among = [&](int r, int first, int last) { return r >= first && r <= last; };
        const bool own_a = among(2 * t, 4, tr - 5), own_b = among(2 * t + 1, 4, tr - 5);
        const DuoTest test{among(2 * t, 0, tr - 1),     among(2 * t + 1, 0, tr - 1), among(2 * t, 2, tr - 3),
                           among(2 * t + 1, 2, tr - 3), among(2 * t, 3, tr - 5),     among(2 * t + 1, 3, tr - 5)};
        if (duo_sweeps<METHOD, SLOPE, FT, 1, TT, 1, false, CYL_NONE, true>(ua, ub, true, p, planes, SS, lambda, c, DuoGeo{}, test)) {
            double xa[5], xb[5];
            fetch(2 * t, xa);
            fetch(2 * t + 1, xb);
            __syncthreads();
            // in line: a call's saved registers cost every chunk more (1500 problems 2.85 against 2.78 ms)
            duo_sweeps<METHOD, SLOPE, FT, 1, TT, 1, false, CYL_NONE, true, WideOps>(xa, xb, true, p, planes, SS, lambda, c, DuoGeo{});
#pragma unroll
            for (int k = 0; k < 5; k++) { ua[k] = xa[k]; ub[k] = xb[k]; }
        }
        // every thread has read this chunk's inputs
        ens_store_pending(qb, S, ch, cb, t, pend);
        if (own_a) ens_store(qb, S, ch, cb, len, single, 2 * t - 4, ua, pend, first);
        if (own_b) ens_store(qb, S, ch, cb, len, single, 2 * t - 3, ub, pend, first);
    }
    ens_store_ends(qb, S, n, nchunks, t, pend, first);
}

// One row a thread: three CTAs of 256 threads per SM (80 registers) rather than four: at 64 registers a
// thread's state of two stages spills; 512-thread CTAs keep two per SM, one would idle half the SM.
// TWO: two rows a thread, CTAs of half the launch shape's `threads`, per SM as for the row kernel
// (duo_min_blocks): five of 128 threads at 96 registers for the default shape.
template <int METHOD, int SLOPE, typename FT, int NT, bool TWO>
__global__ void __launch_bounds__(TWO ? NT / 2 : NT,
                                  TWO ? (NT == 128 ? 2 * duo_min_blocks<FT>(128) : duo_min_blocks<FT>(NT / 2))
                                      : (NT == 512 ? 2 : 768 / NT)) ensemble_kernel(EnsArgs a, FluidConsts<FT> c)
{
    extern __shared__ __align__(16) double tsm[];
    __shared__ int s_prob;
    constexpr int TT = TWO ? NT / 2 : NT;
    __shared__ double s_red[TT / 32];
    __shared__ double s_dt;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *pend = tsm;        // [2][5][4]
    double *first = tsm + 40;  // [5][4]
    for (;;) {
        if (tid == 0) {
            const unsigned k = atomicAdd(a.counter, 1u);
            s_prob = (k < (unsigned)a.np) ? (a.order ? a.order[k] : (int)k) : -1;
        }
        __syncthreads();
        const int p = s_prob;
        if (p < 0) break;
        const int64_t off = a.off[p];
        const int64_t nn = a.off[p + 1] - off;
        const double h = a.h[p];
        const int n = (int)nn;
        const int nc = (nn >= 9 && nn < (1 << 30)) ? ens_nchunks(n, a.target) : 0;
        if (nc == 0 || (n + nc - 1) / nc + 8 > a.lcap || p >= a.np) {
            if (tid == 0 && p < a.np) {
                a.t_out[p] = 0.0;
                a.it_out[p] = -1;  // not run: fewer than 9 cells or a chunk beyond the tile
            }
            __syncthreads();
            continue;
        }
        double *qb = a.q + off;
        double t = 0.0, kc = 0.0;
        int it = 0;
        while (it < a.itermax && t < a.t_end * (1 - 1e-14)) {
            // tau: NaN-ignoring minimum of the signal-crossing times, halved for HLL/HLLC
            double tmin = 1e37;
            for (int x = tid; x < n; x += TT) {
                const double rho = qb[x], px = qb[x + 2 * a.S];
                const double cs = soundspeed_cell(rho, qb[x + a.S], px, qb[x + 3 * a.S], qb[x + 4 * a.S], a.gg1);
                tmin = min_keep(tmin, cfl_cell<1, false>(rho, px, 0.0, 0.0, cs, h, h, h, h));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tmin = min_keep(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
            if (lane == 0) s_red[wid] = tmin;
            __syncthreads();
            if (tid == 0) {
                double r = 1e38;
                for (int w = 0; w < TT / 32; w++) r = (s_red[w] < r) ? s_red[w] : r;
                if (a.halve) r = r / 2;
                double dt = __dmul_rn(a.cfl, r);
                if (__dadd_rn(t, __dmul_rn(2.0, dt)) > a.t_end) dt = __dmul_rn(.5, __dadd_rn(a.t_end, -t));
                s_dt = dt;
            }
            __syncthreads();
            const double dt = s_dt;
            const double lambda = dt / h;
            for (int half = 0; half < 2; half++) {
                if constexpr (TWO) {
                    double *SS = tsm + 60;  // the SSPRK sums, then the planes
                    ens_sweep_two<METHOD, SLOPE, FT, TT>(qb, a.S, n, nc, lambda, c,
                                                         reinterpret_cast<FT *>(SS + 10 * TT), SS, pend, first);
                } else {
                    FT *SA = reinterpret_cast<FT *>(tsm + 60);  // [5][lcap]
                    ens_sweep<METHOD, SLOPE, FT, NT>(qb, a.S, n, nc, lambda, c, SA, SA + 5 * a.lcap, a.lcap, pend, first);
                }
                if (tid == 0) ens_boundary(qb, a.S, n, a.bc0, a.bc1);
                __syncthreads();
            }
            const double y = __dadd_rn(__dmul_rn(2.0, dt), -kc);
            const double tn = __dadd_rn(t, y);
            kc = __dadd_rn(__dadd_rn(tn, -t), -y);
            t = tn;
            it++;
        }
        if (tid == 0) {
            a.t_out[p] = t;
            a.it_out[p] = it;
        }
        __syncthreads();
    }
}

// Shared memory of one CTA: the pending and first outputs, and two planes of a chunk of up to lcap tile
// rows, or the sums and planes of two rows a thread.
template <typename FT, int NT, bool TWO>
static size_t ens_smem(int lcap)
{
    return sizeof(double) * 60 + (TWO ? duo_smem_bytes<FT, NT / 2>() : sizeof(FT) * 10 * (size_t)lcap);
}

template <int METHOD, int SLOPE, typename FT, int NT, bool TWO>
static int launch_ens_nt(const EnsArgs &a0, const FluidConsts<FT> &c, int ctas_per_sm, cudaStream_t st)
{
    EnsArgs a = a0;
    auto kern = ensemble_kernel<METHOD, SLOPE, FT, NT, TWO>;
    constexpr int TT = TWO ? NT / 2 : NT;
    const size_t shm = ens_smem<FT, NT, TWO>(a.lcap);
    static SmemOptIn record;
    int rc;
    if ((rc = opt_in(record, kern, shm))) return rc;
    int per_sm = 0;
    if ((rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TT, shm)))) return rc;
    if (per_sm < 1 || a.lcap > NT) return IB_ERROR_INVALID_ARGS;
    // a CTA of two rows a thread counts as half a CTA of the launch shape's `threads`, so that a limit keeps
    // the rows in flight that it was chosen for
    const int limit = TWO ? 2 * ctas_per_sm : ctas_per_sm;
    if (limit > 0 && limit < per_sm) per_sm = limit;
    const int64_t grid = std::min<int64_t>((int64_t)per_sm * num_sms(), a.np);
    if ((rc = check_cuda(cudaMemsetAsync(a.counter, 0, sizeof(unsigned int), st)))) return rc;
    kern<<<(unsigned)grid, TT, shm, st>>>(a, c);
    return check_launch();
}

// Two rows a thread from nine problems per SM on: half the shared-memory traffic, but a CTA of half the threads takes
// longer for a problem, and with fewer problems a problem's own time counts.  Time against one row a thread:
//   problems                        600    900    1100   1300   1480   2000   3000
//   FP64, 256-4096 cells            1.31   1.34   1.14   0.97   0.94   0.95   0.95
//   FP64, 32-512 cells              1.44   1.20   1.07   0.99   0.97   0.97   0.98
//   FP64, 900-1100 cells            0.98   1.12   1.08   0.98   0.95   0.95   0.99
//   FP32 flux, 256-4096 cells       1.13   1.38   1.17   1.00   0.90   0.80   0.79
//   FP32 flux, 32-512 cells         1.23   1.18   1.04   0.96   0.83   0.82   0.80
//   FP32 flux, 900-1100 cells       0.92   0.85   0.93   0.83   0.84   0.84   0.80
// (FP64 256-4096 cells, 10 iterations: 1480 problems 3.00 -> 2.81 ms, 3000 5.89 -> 5.59; FP32 flux 2.35 -> 2.11, 4.62 ->
// 3.62).  By the number of problems and SMs alone: both forms give the same bits.
static bool ens_two_rows(int np) { return np >= 9 * num_sms(); }

template <int METHOD, int SLOPE, typename FT, int NT>
static int launch_ens_form(const EnsArgs &a, const FluidConsts<FT> &c, int ctas_per_sm, cudaStream_t st)
{
    return ens_two_rows(a.np) ? launch_ens_nt<METHOD, SLOPE, FT, NT, true>(a, c, ctas_per_sm, st)
                              : launch_ens_nt<METHOD, SLOPE, FT, NT, false>(a, c, ctas_per_sm, st);
}

template <int METHOD, int SLOPE, typename FT>
static int launch_ens(const EnsArgs &a, const FluidConsts<FT> &c, int threads, int ctas_per_sm, cudaStream_t st)
{
    switch (threads) {
    case 128: return launch_ens_form<METHOD, SLOPE, FT, 128>(a, c, ctas_per_sm, st);
    case 256: return launch_ens_form<METHOD, SLOPE, FT, 256>(a, c, ctas_per_sm, st);
    case 512: return launch_ens_form<METHOD, SLOPE, FT, 512>(a, c, ctas_per_sm, st);
    default: return IB_ERROR_INVALID_ARGS;
    }
}

template <int METHOD, typename FT>
static int launch_ens_slope(int slope, const EnsArgs &a, const FluidConsts<FT> &c, int threads, int cps,
                            cudaStream_t st)
{
    if (slope == IB_SLOPE_MC) return launch_ens<METHOD, IB_SLOPE_MC, FT>(a, c, threads, cps, st);
    if (slope == IB_SLOPE_OSPRE) return launch_ens<METHOD, IB_SLOPE_OSPRE, FT>(a, c, threads, cps, st);
    return IB_ERROR_NOIMPLEMENT;
}

}  // namespace ib

using namespace ib;

extern "C" int ib_riemannEnsemble(const ib_ensemble *e, const ib_fluid_thermo *thermo, int method, double cfl,
                                  double t_end, int32_t itermax, const ib_numerics *num,
                                  const ib_ensemble_tuning *tuning, void *stream)
{
    if (!e || !thermo) return IB_ERROR_NULL_POINTER;
    if (!e->q || !e->offsets || !e->h || !e->t_out || !e->iters_out) return IB_ERROR_NULL_POINTER;
    if (e->nproblems < 1 || e->slab_pitch < 1) return IB_ERROR_INVALID_ARGS;
    if (method != IB_METHOD_HLL && method != IB_METHOD_HLLC) return IB_ERROR_NOIMPLEMENT;
    if (!(cfl > 0) || !(t_end >= 0) || !(t_end < 1e300)) return IB_ERROR_INVALID_ARGS;
    for (int s = 0; s < 2; s++) {
        const int m = e->bc[s];
        if (m != IB_BC_CIRCULAR && m != IB_BC_MIRROR && m != IB_BC_CONST && m != IB_BC_LINEAR && m != IB_BC_OUTFLOW)
            return IB_ERROR_INVALID_ARGS;
    }
    const double gamma = thermo->gamma;
    if (!(gamma > 1)) return IB_ERROR_INVALID_ARGS;
    if (thermo->c_isothermal != -1) return IB_ERROR_NOIMPLEMENT;
    const int slope = num ? num->slope_limiter : IB_SLOPE_OSPRE;
    const int prec = num ? num->precision : IB_PREC_FP64;
    int threads = 256, chunk = 0, cps = 0;
    if (tuning) {
        if (tuning->threads) threads = tuning->threads;
        chunk = tuning->chunk;
        cps = tuning->ctas_per_sm;
    }
    if (threads != 128 && threads != 256 && threads != 512) return IB_ERROR_INVALID_ARGS;
    if (chunk == 0) chunk = threads - 8;
    if (chunk < 120 || chunk > threads - 8 || cps < 0) return IB_ERROR_INVALID_ARGS;
    EnsArgs a;
    a.q = e->q;
    a.S = e->slab_pitch;
    a.off = e->offsets;
    a.h = e->h;
    a.order = e->order;
    a.t_out = e->t_out;
    a.it_out = e->iters_out;
    a.counter = scratch().ensemble_counter();
    if (!a.counter) return IB_ERROR_NOMEM;
    a.np = e->nproblems;
    a.bc0 = e->bc[0];
    a.bc1 = e->bc[1];
    a.itermax = (itermax > 0) ? itermax : 0x7fffffff;
    a.target = chunk;
    a.lcap = chunk + 8;
    a.gg1 = gamma * (gamma - 1);
    a.cfl = cfl;
    a.t_end = t_end;
    a.halve = 1;
    cudaStream_t st = (cudaStream_t)stream;
    const double rho_min = thermo->rho_min;
    if (method == IB_METHOD_HLLC) {
        if (prec == IB_PREC_FP32_FLUX)
            return launch_ens_slope<IB_METHOD_HLLC, float>(slope, a, make_consts<float>(gamma, rho_min, -1), threads,
                                                          cps, st);
        if (prec != IB_PREC_FP64) return IB_ERROR_INVALID_ARGS;
        return launch_ens_slope<IB_METHOD_HLLC, double>(slope, a, make_consts<double>(gamma, rho_min, -1), threads,
                                                       cps, st);
    }
    if (prec != IB_PREC_FP64) return IB_ERROR_NOIMPLEMENT;
    return launch_ens_slope<IB_METHOD_HLL, double>(slope, a, make_consts<double>(gamma, rho_min, -1), threads, cps,
                                                  st);
}
