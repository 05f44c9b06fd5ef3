// ib_duo.cuh -- sweep kernels with two neighbouring cells a thread: x rows of up to 1024 cells, and y/z
// pencils of up to 512 cells that TMA cannot fetch (odd nx, unaligned arrays).
//
// A thread owns the cells a = 2t and b = 2t + 1 and a CTA whole pencils, so that both SSPRK stages run on
// chip (ib_sweep.cuh).  What bounds such a sweep, once its divisions and square roots are the short ones of
// ib_fast.cuh, is the traffic between threads through shared memory: with one cell a thread the data pipe was
// 70 % busy in the 256^3 x sweep.  Two cells a thread exchange only b's primitives with the thread after and
// a's with the one before, one face and one flux: half the bytes per cell (data pipe 50 %), no exchange at all
// for the face between a and b, and two independent chains of FP64 arithmetic (256^3 HLLC x 0.534 -> 0.461 ms
// at five 128-thread CTAs of 96 registers per SM; 128 registers and four CTAs 0.483, 80 and six 0.565 with
// spills).  The y/z boxes that TMA fetches stay with the one-cell kernels: there the wait for a box weighs more
// than the exchange, and the fewer warps of this form hide it less (256^3 y: 0.552 against 0.580 ms).
//
// Per stage: primitives to shared memory, barrier, limited slopes, the flux through a|b and a's left
// face to shared memory, barrier, the flux through b's right face to shared memory, barrier, update.
// (Forming the right neighbour's face again instead of exchanging it saves a barrier but measured slower,
// 0.461 -> 0.492 ms: more live registers.)  Three planes of 5 x TT values rotate through the roles
// (primitives of a, later fluxes; primitives of b; left faces) so that no stage writes a plane which the one
// before may still be reading.
#pragma once

#include "ib_bc.cuh"
#include "ib_sweep.cuh"

namespace ib {

// A thread's place: plane slots of its own cells, of the thread before and the one after (periodic).
// Pencils of odd length: the last thread owns only a; its b stands for the pencil's first cell.
struct DuoPos {
    int own, left, right;
    bool first, ghost;  // odd lengths only: the pencil's first thread, the last one
};

struct DuoGeo {
    double ra, rb, dr;  // radial sweeps: the radii of the two cells' centres, the cell size
    double rpen;        // theta sweeps: the pencil's radius
};

// What of a thread's two cells is tested for operands that the short forms do not reach, in the last sweep: the
// primitives of the first stage (in), those of the second (mid), the second stage's mass flux through the cell's
// right face (face).  A CTA of whole pencils tests the last two of each of its cells.  One that works on part of a
// pencil tests `face` at the faces of the cells that it returns, `mid` where the second stage's input is theirs to use,
// and `in` of every cell it loaded: a limiter can drop the NaN of a cell beyond.
struct DuoTest {
    bool in_a, in_b, mid_a, mid_b, face_a, face_b;
};

// NS sweeps of the cells (ua, ub) of this thread, in place.  planes: 15 TT values of FT; SS: 10 TT
// doubles, where u1 + u0 of the SSPRK average waits through the second stage.  All threads of the CTA
// call it.  OPS: FastOps (returns to all threads whether a test of theirs asks for the sweep to be done again, with
// the inputs of old) or IeeeOps.
template <int METHOD, int SLOPE, typename FT, int DIR, int TT, int NS, bool ODD, int GEO, bool RN = false,
          typename OPS = FastOps>
__device__ __forceinline__ bool duo_sweeps(double (&ua)[5], double (&ub)[5], bool act, const DuoPos &p, FT *planes,
                                           double *SS, double lambda, const FluidConsts<FT> &c, const DuoGeo &g,
                                           const DuoTest &test = DuoTest{})
{
    double va[5], vb[5];
    bool suspect = false;
#pragma unroll
    for (int s = 0; s < 2 * NS; s++) {
        const bool second = s & 1;
        FT *P = planes + (s % 3) * 5 * TT, *Q = planes + ((s + 1) % 3) * 5 * TT, *R = planes + ((s + 2) % 3) * 5 * TT;
        V5<FT> wa, wb;
        if (act) {
            wa = stage_prims<METHOD, DIR, FT, RN, OPS>(second ? va : ua, c);  // HLL floors its argument
            wb = stage_prims<METHOD, DIR, FT, RN, OPS>(second ? vb : ub, c);
            if constexpr (kPoison<OPS, FT>) {
                if (s == 2 * NS - 2) suspect = (test.in_a && cell_suspect(ua[0], wa.a[3])) || (test.in_b && cell_suspect(ub[0], wb.a[3]));
                if (s == 2 * NS - 1)
                    suspect = suspect || (test.mid_a && cell_suspect(va[0], wa.a[3])) || (test.mid_b && cell_suspect(vb[0], wb.a[3]));
            }
#pragma unroll
            for (int k = 0; k < 5; k++) {
                P[k * TT + p.own] = wa.a[k];
                Q[k * TT + p.own] = wb.a[k];
                if (second) {  // after the prims: HLL floors the stage's input
                    SS[k * TT + p.own] = va[k] + ua[k];
                    SS[(5 + k) * TT + p.own] = vb[k] + ub[k];
                }
            }
        }
        __syncthreads();
        V5<FT> fm, rb;  // the flux through a|b, b's right face
        double pa = 0.0, pb = 0.0;  // radial sweeps: the cells' face pressure sums (HLLC) or input pressures (HLL)
        if (act) {
            V5<FT> lb, ra;
            if (ODD && p.ghost) {
#pragma unroll
                for (int k = 0; k < 5; k++) wb.a[k] = P[k * TT + p.right];
            }
            if (GEO == CYL_RADIAL && METHOD == IB_METHOD_HLL) { pa = (double)wa.a[2]; pb = (double)wb.a[2]; }
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const FT wl = (ODD && p.first) ? P[k * TT + p.left] : Q[k * TT + p.left];
                const FT wr = (ODD && p.ghost) ? Q[k * TT + p.right] : P[k * TT + p.right];
                const FT dl = wa.a[k] - wl, dm = wb.a[k] - wa.a[k], dr = wr - wb.a[k];
                const FT ha = slope_limit<SLOPE, FT, OPS>(dl, dm), hb = slope_limit<SLOPE, FT, OPS>(dm, dr);
                FT la;
                if (METHOD == IB_METHOD_HLLC && k == 1) {  // internal energy to pressure
                    la = product<RN>(c.gm1, wa.a[k] - ha);
                    ra.a[k] = product<RN>(c.gm1, wa.a[k] + ha);
                    lb.a[k] = product<RN>(c.gm1, wb.a[k] - hb);
                    rb.a[k] = product<RN>(c.gm1, wb.a[k] + hb);
                    if (GEO == CYL_RADIAL) {
                        pa = (double)la + (double)ra.a[k];
                        pb = (double)lb.a[k] + (double)rb.a[k];
                    }
                } else {
                    la = wa.a[k] - ha;
                    ra.a[k] = wa.a[k] + ha;
                    lb.a[k] = wb.a[k] - hb;
                    rb.a[k] = wb.a[k] + hb;
                }
                R[k * TT + p.own] = la;
            }
            fm = stage_flux<METHOD, FT, RN, OPS>(c, ra, lb);
        }
        __syncthreads();
        V5<FT> fb;
        if (act) {
            V5<FT> lr;
#pragma unroll
            for (int k = 0; k < 5; k++) lr.a[k] = R[k * TT + p.right];
            fb = stage_flux<METHOD, FT, RN, OPS>(c, rb, lr);
#pragma unroll
            for (int k = 0; k < 5; k++) P[k * TT + p.own] = (ODD && p.ghost) ? fm.a[k] : fb.a[k];
        }
        if (kPoison<OPS, FT> && s == 2 * NS - 1) {
            if (act) suspect = suspect || (test.face_a && fm.a[0] != fm.a[0]) || (test.face_b && fb.a[0] != fb.a[0]);
            suspect = __syncthreads_or(suspect);
        } else {
            __syncthreads();
        }
        if (act) {
            const double lam = (GEO == CYL_THETA_LAM) ? lambda / g.rpen : lambda;
            // the isothermal HLL radial term's density: the new prediction (first stage), the stage's own
            // floored input (second)
            const double rho_a = va[0], rho_b = vb[0];
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const double fl = (double)P[k * TT + p.left], fc = (double)fm.a[k], fr = (double)fb.a[k];
                const double ta = second ? SS[k * TT + p.own] : ua[k], tb = second ? SS[(5 + k) * TT + p.own] : ub[k];
                double na, nb;
                if constexpr (GEO == CYL_NONE) {
                    na = sub_product(ta, lambda, fc - fl);
                    nb = sub_product(tb, lambda, fr - fc);
                } else {
                    na = ta - cyl_dflux<METHOD, GEO>(k, fc, fl, lam, g.ra, g.dr, g.rpen, pa, pa,
                                                     second ? rho_a : (k == 0 ? 0.0 : va[0]), c);
                    nb = tb - cyl_dflux<METHOD, GEO>(k, fr, fc, lam, g.rb, g.dr, g.rpen, pb, pb,
                                                     second ? rho_b : (k == 0 ? 0.0 : vb[0]), c);
                }
                if (second) {
                    ua[k] = .5 * na;
                    ub[k] = .5 * nb;
                } else {
                    va[k] = na;
                    vb[k] = nb;
                }
            }
        }
    }
    return suspect;
}

// The same with the IEEE operations, out of line: its registers are not the caller's.
template <int METHOD, int SLOPE, typename FT, int DIR, int TT, bool RN>
__device__ __noinline__ void duo_sweep_ieee(double (&ua)[5], double (&ub)[5], DuoPos p, FT *planes, double *SS, double lambda,
                                            FluidConsts<FT> c)
{
    duo_sweeps<METHOD, SLOPE, FT, DIR, TT, 1, false, CYL_NONE, RN, IeeeOps>(ua, ub, true, p, planes, SS, lambda, c, DuoGeo{});
}

// Dynamic shared memory of a CTA of TT threads: the planes and the SSPRK sums.
template <typename FT, int TT>
__host__ __device__ constexpr size_t duo_smem_bytes() { return (size_t)15 * TT * sizeof(FT) + (size_t)80 * TT; }

// CTAs per SM that the registers are held to: about 20 warps of 96 registers per SM for FP64, 24 of 80 for the
// FP32 flux (256^3 x: 0.327 ms against 0.352 at 96); FP64 CTAs of 256 and 512 threads take 128 registers
template <typename FT>
constexpr int duo_min_blocks(int TT)
{
    if (sizeof(FT) == 4) return TT <= 128 ? 6 : (TT <= 160 ? 5 : (TT <= 192 ? 4 : (TT <= 256 ? 3 : 1)));
    return TT <= 128 ? 5 : (TT <= 160 ? 4 : (TT <= 192 ? 3 : (TT <= 256 ? 2 : 1)));
}

// ------------------------------------------------------------------------------------------
// x rows: rp rows per CTA (short rows share one), T = ceil(n / 2) threads each.  vec: 16-byte accesses.
// FILL: the fill of the rows' ends follows, from the stored rows (a launch of its own took 2.3 us).  Its own
// instantiation: the values it keeps to the end spill in the sweep (256^3 x 0.469 -> 0.483 ms with a run-time
// test).
// ------------------------------------------------------------------------------------------
template <int METHOD, int SLOPE, typename FT, int TT, int NS, bool ODD, bool FILL, int GEO>
__global__ void __launch_bounds__(TT, duo_min_blocks<FT>(TT)) duo_row_kernel(SweepArgs a, FluidConsts<FT> c, int rp, int T, int vec)
{
    extern __shared__ __align__(16) unsigned char row_smem_raw[];
    double *SS = reinterpret_cast<double *>(row_smem_raw);
    FT *planes = reinterpret_cast<FT *>(SS + 10 * TT);
    if (a.lambda.off()) return;  // a device timestep of 0: after the end time
    const double lambda = a.lambda.get();
    const int n = a.nx;
    const int r = threadIdx.x / T, t = threadIdx.x - r * T;
    const int64_t row = (int64_t)blockIdx.x * rp + r;
    const bool act = r < rp && row < (int64_t)a.ny * a.nz;
    DuoPos p;
    p.own = threadIdx.x;
    p.left = (t == 0) ? p.own + T - 1 : p.own - 1;
    p.right = (t == T - 1) ? p.own - (T - 1) : p.own + 1;
    p.first = ODD && t == 0;
    p.ghost = ODD && t == T - 1;
    double ua[5], ub[5];
    double *q = a.q + row * n + 2 * t;
#pragma unroll
    for (int k = 0; k < 5; k++) ua[k] = ub[k] = 1.0;
    if (act) {
        if (!ODD && vec) {
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const double2 v = *reinterpret_cast<const double2 *>(q + (int64_t)slot_of<METHOD, 1>(k) * a.slab);
                ua[k] = v.x;
                ub[k] = v.y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 5; k++) {
                ua[k] = q[(int64_t)slot_of<METHOD, 1>(k) * a.slab];
                if (!p.ghost) ub[k] = q[(int64_t)slot_of<METHOD, 1>(k) * a.slab + 1];
            }
        }
    }
    DuoGeo g;
    if (GEO == CYL_RADIAL) { g.ra = a.crin + (2 * t) * a.cdr; g.rb = a.crin + (2 * t + 1) * a.cdr; g.dr = a.cdr; }
    const bool whole = !(ODD && p.ghost);  // the last thread of an odd pencil owns one cell
    const bool suspect = duo_sweeps<METHOD, SLOPE, FT, 1, TT, NS, ODD, GEO>(ua, ub, act, p, planes, SS, lambda, c, g,
                                                                           DuoTest{false, false, true, whole, true, whole});
    if (suspect) {
        __syncthreads();  // every thread is done with the planes
        if constexpr (kPoison<FastOps, FT>)
            ieee_pencils<METHOD, SLOPE, 1, GEO>(
                IeeePencils{a.q, a.slab, a.nx, a.ny, a.nz, (int64_t)blockIdx.x * rp, rp, NS, lambda, CylPencil{a.crin, a.cdr, 0, 0}}, c, SS);
    } else if (act) {
        if (!ODD && vec) {
#pragma unroll
            for (int k = 0; k < 5; k++)
                *reinterpret_cast<double2 *>(q + (int64_t)slot_of<METHOD, 1>(k) * a.slab) = make_double2(ua[k], ub[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 5; k++) {
                q[(int64_t)slot_of<METHOD, 1>(k) * a.slab] = ua[k];
                if (!p.ghost) q[(int64_t)slot_of<METHOD, 1>(k) * a.slab + 1] = ub[k];
            }
        }
    }
    if constexpr (FILL) {
        __syncthreads();
        for (int it = threadIdx.x; it < 10 * rp; it += blockDim.x) {
            const int64_t fr = (int64_t)blockIdx.x * rp + it / 10;
            if (fr < (int64_t)a.ny * a.nz) fill_item(a.q + fr * a.nx, a.slab, 1, a.nx, a.bc, 1, it % 10);
        }
    }
}

// ------------------------------------------------------------------------------------------
// y and z pencils by plain loads and stores: COLS pencils per CTA, T = ceil(n / 2) threads each, the
// pencil fastest, so that COLS lanes read neighbouring doubles.
// ------------------------------------------------------------------------------------------
template <int METHOD, int SLOPE, typename FT, int DIR, int TT, int COLS, bool ODD, int GEO>
__global__ void __launch_bounds__(TT, duo_min_blocks<FT>(TT))
    duo_pencil_kernel(SweepArgs a, FluidConsts<FT> c, int64_t npencil, CylPencil cyl)
{
    extern __shared__ __align__(16) unsigned char row_smem_raw[];
    double *SS = reinterpret_cast<double *>(row_smem_raw);
    FT *planes = reinterpret_cast<FT *>(SS + 10 * TT);
    if (a.lambda.off()) return;  // a device timestep of 0: after the end time
    const double lambda = a.lambda.get();
    const PencilMap pm{a.nx, a.ny, a.nz, DIR};
    const int T = (pm.length() + 1) / 2;
    const int t = threadIdx.x / COLS;
    const int64_t pencil = (int64_t)blockIdx.x * COLS + threadIdx.x % COLS;
    const bool act = t < T && pencil < npencil;
    DuoPos p;
    p.own = threadIdx.x;
    p.left = (t == 0) ? p.own + (T - 1) * COLS : p.own - COLS;
    p.right = (t == T - 1) ? p.own - (T - 1) * COLS : p.own + COLS;
    p.first = ODD && t == 0;
    p.ghost = ODD && t == T - 1;
    double *q = a.q + pm.base(pencil) + 2 * t * pm.stride();
    double ua[5], ub[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        ua[k] = act ? q[(int64_t)slot_of<METHOD, DIR>(k) * a.slab] : 1.0;
        ub[k] = (act && !p.ghost) ? q[(int64_t)slot_of<METHOD, DIR>(k) * a.slab + pm.stride()] : 1.0;
    }
    DuoGeo g;
    if (GEO != CYL_NONE) g.rpen = theta_radius(cyl, (int)(pencil % a.nx), (int)(pencil / a.nx));
    const bool whole = !(ODD && p.ghost);
    const bool suspect = duo_sweeps<METHOD, SLOPE, FT, DIR, TT, 1, ODD, GEO>(ua, ub, act, p, planes, SS, lambda, c, g,
                                                                            DuoTest{false, false, true, whole, true, whole});
    if (suspect) {
        __syncthreads();  // every thread is done with the planes
        if constexpr (kPoison<FastOps, FT>)
            ieee_pencils<METHOD, SLOPE, DIR, GEO>(
                IeeePencils{a.q, a.slab, a.nx, a.ny, a.nz, (int64_t)blockIdx.x * COLS, COLS, 1, lambda, cyl}, c, SS);
    } else if (act) {
#pragma unroll
        for (int k = 0; k < 5; k++) {
            q[(int64_t)slot_of<METHOD, DIR>(k) * a.slab] = ua[k];
            if (!p.ghost) q[(int64_t)slot_of<METHOD, DIR>(k) * a.slab + pm.stride()] = ub[k];
        }
    }
}

// ------------------------------------------------------------------------------------------
// Chunks of long pencils (ib_sweep.cuh: jobs, side buffer, tiles): R / 2 threads per column, two rows each.
// ------------------------------------------------------------------------------------------
template <int METHOD, int SLOPE, typename FT, int DIR, int W, int R>
__global__ void __launch_bounds__(R *W / 2, 512 / (R * W / 2))
    sweep_chunk_kernel(const __grid_constant__ CUtensorMap tm, ChunkArgs a, FluidConsts<FT> c)
{
    constexpr int L = R - 8;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[2];
    constexpr size_t tb = ((size_t)40 * L * W + 127) / 128 * 128;
    constexpr size_t hb = ((size_t)320 * W + 127) / 128 * 128;
    // tile and halo block of buffer b (computed, not indexed arrays, which would live in local memory)
    auto Ub = [&](int b) { return reinterpret_cast<double *>(smem_raw + b * tb); };
    auto Hb = [&](int b) { return reinterpret_cast<double *>(smem_raw + 2 * tb + b * hb); };
    double *SS = reinterpret_cast<double *>(smem_raw + 2 * tb + 2 * hb);
    FT *planes = reinterpret_cast<FT *>(smem_raw + 2 * tb + 2 * hb + (size_t)40 * R * W);
    constexpr uint32_t tile_tx = 40u * L * W + 320u * W;
    constexpr int s0 = slot_of<METHOD, DIR>(0), s1 = slot_of<METHOD, DIR>(1), s2 = slot_of<METHOD, DIR>(2),
                  s3 = slot_of<METHOD, DIR>(3), s4 = slot_of<METHOD, DIR>(4);
    const int slots[5] = {s0, s1, s2, s3, s4};
    constexpr int TT = R * W / 2, T = R / 2;
    const int col = (W == 1) ? 0 : (int)(threadIdx.x % W);
    const int t = (int)(threadIdx.x / W);  // this thread's cells: rows 2t and 2t + 1 of the job
    DuoPos p;
    p.own = threadIdx.x;
    p.left = (t > 0) ? p.own - W : p.own;  // the job's edge rows: unused results
    p.right = (t < T - 1) ? p.own + W : p.own;
    p.first = p.ghost = false;
    const int n = a.n, C = a.C;
    if (a.lambda.off()) return;  // a device timestep of 0: after the end time
    const double lambda = a.lambda.get();
    const bool leader = threadIdx.x == 0;
    const int64_t njobs_all = a.ngroups * C;
    const int64_t step = gridDim.x;

    if (leader) {
        prefetch_tmap(&tm);
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int64_t j, int buf) {  // leader only
        mbar_arrive_expect_tx(&full[buf], tile_tx);
        chunk_load<DIR>(Ub(buf), &tm, j / C, (int)(j % C) * L, a, W, &full[buf]);
        bulk_load(Hb(buf), a.side + j * 40 * W, 320u * W, &full[buf]);
    };
    // bit b: a load into buffer b is in flight (leader's bookkeeping) / parity to wait for on b
    uint32_t issued = 0, phase = 0;
    if (leader) {
        for (int t = 0; t < 2; t++) {
            const int64_t jt = blockIdx.x + t * step;
            if (jt < njobs_all) { issue(jt, t); issued |= 1u << t; }
        }
    }
    int it = 0;
    for (int64_t j = blockIdx.x; j < njobs_all; j += step, it++) {
        const int buf = it & 1;
        const int64_t grp = j / C;
        const int cc = (int)(j % C);
        const int c0 = cc * L;                    // first cell of the chunk
        const int cend = (c0 + L < n) ? c0 + L : n;
        const bool ok = mbar_wait_cta(&full[buf], (phase >> buf) & 1, a.spin);
        if (!ok) {
            if (leader) {
                atomicOr(a.err, 1u);
                mbar_wait(&full[buf], (phase >> buf) & 1);  // one more bounded wait for the late tile
                if ((issued >> (buf ^ 1)) & 1) mbar_wait(&full[buf ^ 1], (phase >> (buf ^ 1)) & 1);
            }
            return;
        }
        phase ^= 1u << buf;
        issued &= ~(1u << buf);
        // row r is cell g = c0 - 4 + r: left halo (side buffer), chunk (tile), right halo (side buffer), or
        // idle
        const double *Ut = Ub(buf), *H = Hb(buf);
        auto fetch = [&](int r, double (&u)[5]) {
            const int g = c0 - 4 + r;
            if (g >= c0 && g < cend) {
#pragma unroll
                for (int k = 0; k < 5; k++) u[k] = Ut[(slots[k] * L + (g - c0)) * W + col];
            } else if (g < cend + 4) {
                const int rr = (g < c0) ? r : 4 + (g - cend);
#pragma unroll
                for (int k = 0; k < 5; k++) u[k] = H[(slots[k] * 8 + rr) * W + col];
            } else {
#pragma unroll
                for (int k = 0; k < 5; k++) u[k] = 1.0;
            }
        };
        double ua[5], ub[5];
        fetch(2 * t, ua);
        fetch(2 * t + 1, ub);
        __syncthreads();  // every thread is done with the planes
        const int g = c0 - 4 + 2 * t;
        const bool own_a = g >= c0 && g < cend, own_b = g + 1 >= c0 && g + 1 < cend;
        const int last = cend - c0 + 7;  // the last row with a cell
        const auto among = [&](int r, int skip) { return r >= skip && r <= last - skip; };
        const DuoTest test{among(2 * t, 0),     among(2 * t + 1, 0),     among(2 * t, 2),
                           among(2 * t + 1, 2), own_a || g == c0 - 1,    own_b || g + 1 == c0 - 1};
        if (duo_sweeps<METHOD, SLOPE, FT, DIR, TT, 1, false, CYL_NONE>(ua, ub, true, p, planes, SS, lambda, c, DuoGeo{}, test)) {
            double xa[5], xb[5];
            fetch(2 * t, xa);
            fetch(2 * t + 1, xb);
            __syncthreads();
            duo_sweep_ieee<METHOD, SLOPE, FT, DIR, TT, false>(xa, xb, p, planes, SS, lambda, c);
#pragma unroll
            for (int k = 0; k < 5; k++) { ua[k] = xa[k]; ub[k] = xb[k]; }
            __syncthreads();
        }
        // every thread is done with tile buf: request the job after next into it
        if (leader) {
            const int64_t jn = j + 2 * step;
            if (jn < njobs_all) {
                fence_proxy_async_smem();
                issue(jn, buf);
                issued |= 1u << buf;
            }
        }
        double *base = a.q + chunk_base(a, DIR, W, grp, col);
#pragma unroll
        for (int k = 0; k < 5; k++) {
            double *cell = base + slots[k] * a.slab + (int64_t)g * a.rs;
            if (own_a) cell[0] = ua[k];
            if (own_b) cell[a.rs] = ub[k];
        }
    }
}

}  // namespace ib
