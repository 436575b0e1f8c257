// k_mg.cu -- multigrid kernels: per-level viscosity, eigenvalue ratios,
// folded 13-point operator, Richardson/Chebyshev sweeps, residual,
// restriction, prolongation and the coarsest-grid banded LU.
//
// Reference: iterative_solver.f90 (multigrid :79-173, prolong :175-233,
// compute_residual :258-279, viscosity_gradients :290-329, compute_viscosity
// :331-377, viscosityBCs(_initialize) :379-453, stream_space :456-561,
// compute_RHS :563-594, restrict(_coefficients) :596-664, test_eigenvalues
// :666-698, iterate_local_time_steps :700-748, eigI/eigR :750-857,
// iterate_stream :860-963, enforceBCs_stream :965-989,
// Compute_Matrix_coarse :1026-1179, Compute_coarse_vector :1181-1193,
// Stream_grid_coarse :1195-1204) and smoother.f90 (vis_space, smoother_vis).
// The kernels specialise the metric terms to the uniform grid (xr=zs=1,
// xrr=...=0), which leaves every retained product and sum of the reference
// unchanged.
#include "tc_cluster.cuh"
#include "tc_device.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#include <stdio.h>

// ---------------------------------------------------------------------------
// visf on the full ghost-padded level-1 box (momentum.f90:1-30; ivis 0,1,2,-1)
// ---------------------------------------------------------------------------
__global__ void k_visf1(Lay L, Phys P, Range2 r, double* __restrict__ vis, const double* __restrict__ Tvis, CPtrs C,
                        const double* __restrict__ zg, const double* __restrict__ T,
                        const double* __restrict__ strain) {
    RANGE_IK(r);
    if (!inr) return;
    size_t x = IX(L, i, k);
    double v;
    if (P.ivis == 1) {
        v = exp(-Tvis[x] * P.lnvisT + (1.0 - zg[k]) * P.lnvisP);
    } else if (P.ivis == 2 && P.comp == 1) {
        double d = 0.0;
        for (int j = 0; j < P.ntype; j++) d = d + C.p[j][x] * P.lnvisC[j];
        if (P.RaT != 0.0) v = exp(-Tvis[x] * P.lnvisT - d + (1.0 - zg[k]) * P.lnvisP);
        else v = exp(-d + (1.0 - zg[k]) * P.lnvisP);
    } else if (P.ivis == 3) {
        // diffusion creep visT**(-T), in parallel with plastic yielding
        // (yield + yield_gradient*z)/strain in the top yield_depth; the
        // strain rate at a ghost node is that of its mirror node
        // (compute_strain_rate_invariant's ghost copies)
        const double diffusion = pow(P.visT, -T[x]);
        const int mi = (i < 0) ? -i : (i > L.a ? 2 * L.a - i : i);
        const int mk = (k < 0) ? -k : (k > L.b ? 2 * L.b - k : k);
        const double sr = strain[IX(L, mi, mk)];
        if (zg[k] < (1.0 - P.yield_depth) || sr == 0.0) {
            v = diffusion;
        } else {
            const double plastic = (P.yield + P.yield_gradient * zg[k]) / sr;
            v = 1.0 / (1.0 / diffusion + 1.0 / plastic);
        }
    } else if (P.ivis == -1) {
        v = exp((1.0 - zg[k]) * P.lnvisP);
    } else {
        v = 1.0;
    }
    vis[x] = v;
}
void launch_visf_level1(cudaStream_t s, const Lay& L, const Phys& P, double* vis, const double* Tvis,
                        const double* const* Cvis, const double* zg, const double* T, const double* strain) {
    Range2 r{-SP, L.a + SP, -SP, L.b + SP};
    CPtrs C{};
    for (int j = 0; j < P.ntype && j < TC_MAX_TYPES; j++) C.p[j] = Cvis[j];
    k_visf1<<<grid_for(r), dim3(BX, BY), 0, s>>>(L, P, r, vis, Tvis, C, zg, T, strain); tc_note_launch();
}

// ---------------------------------------------------------------------------
// viscosity_gradients (+ test_eigenvalues ratio and its minimum)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void eig_pair(const LevConst& c, double v, double vx, double vz, double vxx, double vzz,
                                         double vxz, double& eR, double& eI) {
    double t1 = (vxx - vzz) * c.eK1;
    double t2 = v * c.eK2;
    double t3 = v * (2.0 * c.eTrrss);
    double t4 = vxz * (4.0 * c.eTrs);
    eR = -(t1 + t2 + t3 + t4);
    double t5 = vx * (2.0 * c.eK5);
    double t6 = vz * (2.0 * c.eK6);
    eI = fabs(t5) + fabs(t6);
}

// eigI / eigR of a stretched-grid level at node (i, k) (iterative_solver.f90:
// 750-857), the reference's expressions in its order; the level's node i is
// fine node i * mf
__device__ void eig_pair_metric(const LevConst& c, int i, int k, double v, double vx, double vz, double vxx,
                                double vzz, double vxz, double& eR, double& eI) {
    const int i1 = i * c.mf, k1 = k * c.mf;
    const Metric& M = c.M;
    const double x1 = mt(M.xr, i1), x2 = mt(M.xrr, i1), x3 = mt(M.xrrr, i1), x4 = mt(M.xrrrr, i1);
    const double x13 = mt(M.xr3, i1), x14 = mt(M.xr4, i1);
    const double z1 = mt(M.zs, k1), z2 = mt(M.zss, k1), z3 = mt(M.zsss, k1), z4 = mt(M.zssss, k1);
    const double z13 = mt(M.zs3, k1), z14 = mt(M.zs4, k1);
    const EigScaled& e = c.e;
    {
        const double Sr = e.Tr, Ss = e.Ts, Srr = 0.0, Sss = 0.0, Srrr = e.Trrr, Ssss = e.Tsss, Srrrr = 0.0,
                     Sssss = 0.0, Srs = 0.0, Srrs = e.Trrs, Srss = e.Trss, Srrss = 0.0;
        const double Sx = Sr / x1, Sz = Ss / z1;
        const double Sxx = (Srr + fabs(Sx * x2)) / (x1 * x1);
        const double Szz = (Sss + fabs(Sz * z2)) / (z1 * z1);
        const double Sxxx = (Srrr + fabs(3.0 * Sxx * x1 * x2) + fabs(Sx * x3)) / fabs(x13);
        const double Szzz = (Ssss + fabs(3.0 * Szz * z1 * z2) + fabs(Sz * z3)) / fabs(z13);
        const double Sxxxx =
            (Srrrr + fabs(6.0 * Sxxx * x2 * (x1 * x1)) + (fabs(3.0 * (x2 * x2) + 4.0 * x1 * x3) * fabs(Sxx)) +
             fabs(Sx * x4)) / x14;
        const double Szzzz =
            (Sssss + fabs(6.0 * Szzz * z2 * (z1 * z1)) + (fabs(3.0 * (z2 * z2) + 4.0 * z1 * z3) * fabs(Szz)) +
             fabs(Sz * z4)) / z14;
        const double Sxz = Srs / x1 / z1;
        const double Sxxz = (Srrs + fabs(Sxz * z1 * x2)) / fabs(z1) / (x1 * x1);
        const double Sxzz = (Srss + fabs(Sxz * x1 * z2)) / fabs(x1) / (z1 * z1);
        const double Sxxzz = (Srrss + fabs(Sxzz * x2) * (z1 * z1) + fabs(Sxxz * z2) * (x1 * x1) +
                              fabs(Sxz * x2 * z2)) / ((x1 * z1) * (x1 * z1));
        const double t1 = (vxx + vzz) * (Sxx + Szz);
        const double t2 = v * (Sxxxx + Szzzz);
        const double t3 = 2.0 * v * Sxxzz;
        const double t4 = 4.0 * vxz * Sxz;
        const double t5 = 2.0 * vx * (Sxxx + Sxzz);
        const double t6 = 2.0 * vz * (Szzz + Sxxz);
        eI = fabs(t1) + fabs(t2) + fabs(t3) + fabs(t4) + fabs(t5) + fabs(t6);
    }
    {
        const double q[12] = {0.0, e.Trr, 0.0, e.Trrrr, 0.0, e.Tss, 0.0, e.Tssss, e.Trs, 0.0, 0.0, e.Trrss};
        eR = -stream_op_metric(q, x1, x2, x3, x4, x13, x14, z1, z2, z3, z4, z13, z14, v, vx, vz, vxx, vzz, vxz);
    }
}

// viscosity_gradients' differences, -0.5 vm + 0.5 vp over dr and so on.  The factors that
// are powers of two are exact, so they go into the spacing; half the FP64 operations.
struct VisDiff {
    double r, rr, s, ss, rs;
};
__device__ __forceinline__ VisDiff vis_diff(const LevConst& c, double v0, double vm, double vp, double vzm, double vzp,
                                            double mm, double pm, double mp, double pp) {
    VisDiff d;
    d.r = first_diff(vm, vp, c.dr, c.rdr, c.recip);
    d.rr = spacing_quot(second_diff(vm, v0, vp), c.dr2, c.rdr2, c.recip);
    d.s = first_diff(vzm, vzp, c.ds, c.rds, c.recip);
    d.ss = spacing_quot(second_diff(vzm, v0, vzp), c.ds2, c.rds2, c.recip);
    d.rs = spacing_quot(((mm - pm) - mp) + pp, 4.0 * c.drds, 0.25 * c.rdrds, c.recip);
    return d;
}

// viscosity_gradients at node (i, k) (in d) and, if asked, |eigR / eigI|
template <bool METRIC>
__device__ __forceinline__ double vis_point(const LevConst& c, int i, int k, bool eig, double v0, double vm, double vp,
                                            double vzm, double vzp, double mm, double pm, double mp, double pp,
                                            VisDiff& d) {
    d = vis_diff(c, v0, vm, vp, vzm, vzp, mm, pm, mp, pp);
    double eR = 0.0, eI = 1.0;
    if (METRIC) {
        // viscosity_gradients on a stretched grid (iterative_solver.f90:320-324)
        const int ii = i * c.mf, kk = k * c.mf;
        const double x1 = mt(c.M.xr, ii), x2 = mt(c.M.xrr, ii), z1 = mt(c.M.zs, kk), z2 = mt(c.M.zss, kk);
        const double ax = d.r / x1, az = d.s / z1;
        const double axx = (d.rr - ax * x2) / (x1 * x1), azz = (d.ss - az * z2) / (z1 * z1);
        d.rs = d.rs / x1 / z1;
        d.r = ax; d.s = az; d.rr = axx; d.ss = azz;
        if (eig) eig_pair_metric(c, i, k, v0, d.r, d.s, d.rr, d.ss, d.rs, eR, eI);
    } else if (eig) {
        eig_pair(c, v0, d.r, d.s, d.rr, d.ss, d.rs, eR, eI);
    }
    return eig ? fabs(eR / eI) : 0.0;
}
// vis_space (smoother.f90:142-164): the Laplacian that smooths the viscosity
template <bool METRIC>
__device__ __forceinline__ double vis_laplacian(const LevConst& c, int i, int k, double v0, double vm, double vp,
                                                double vzm, double vzp) {
    const double Trr = spacing_quot(second_diff(vm, v0, vp), c.dr2, c.rdr2, c.recip);
    const double Tss = spacing_quot(second_diff(vzm, v0, vzp), c.ds2, c.rds2, c.recip);
    if (!METRIC) return Trr + Tss;
    const double Tr = first_diff(vm, vp, c.dr, c.rdr, c.recip), Ts = first_diff(vzm, vzp, c.ds, c.rds, c.recip);
    const int i1 = i * c.mf, k1 = k * c.mf;
    const double x1 = mt(c.M.xr, i1), x2 = mt(c.M.xrr, i1), z1 = mt(c.M.zs, k1), z2 = mt(c.M.zss, k1);
    const double Tx = Tr / x1, Tz = Ts / z1;
    const double Txx = (Trr - Tx * x2) / (x1 * x1), Tzz = (Tss - Tz * z2) / (z1 * z1);
    return Txx + Tzz;
}

__global__ void k_vis_grad(Lay L, LevConst c, Range2 r, const double* __restrict__ V, double* __restrict__ vx,
                           double* __restrict__ vz, double* __restrict__ vxx, double* __restrict__ vzz,
                           double* __restrict__ vxz, double* __restrict__ ratio, int do_eig, int ivis,
                           RedScratch rs, double* out_min) {
    RANGE_IK(r);
    double rat = INFINITY;
    if (inr) {
        size_t x = IX(L, i, k);
        if (ivis == 0) {
            vx[x] = 0.0; vz[x] = 0.0; vxx[x] = 0.0; vzz[x] = 0.0; vxz[x] = 0.0;
        } else {
            const size_t ld = (size_t)L.ld;
            const double v0 = V[x], vm = V[x - 1], vp = V[x + 1], vzm = V[x - ld], vzp = V[x + ld];
            const double mm = V[x - 1 - ld], pm = V[x + 1 - ld], mp = V[x - 1 + ld], pp = V[x + 1 + ld];
            VisDiff d;
            rat = c.M.on ? vis_point<true>(c, i, k, do_eig != 0, v0, vm, vp, vzm, vzp, mm, pm, mp, pp, d)
                         : vis_point<false>(c, i, k, do_eig != 0, v0, vm, vp, vzm, vzp, mm, pm, mp, pp, d);
            vx[x] = d.r; vz[x] = d.s; vxx[x] = d.rr; vzz[x] = d.ss; vxz[x] = d.rs;
            if (do_eig) ratio[x] = rat;
        }
    }
    if (do_eig && ivis != 0) reduce_to(RED_MIN, rat, rs.part, rs.count, out_min);
}
void launch_vis_grad(cudaStream_t s, const Level& lv, const double* vis, int do_eig, int ivis, RedScratch rs,
                     DevScalars* ds) {
    Range2 r{1, lv.L.a - 1, 1, lv.L.b - 1};
    k_vis_grad<<<grid_for(r), dim3(BX, BY), 0, s>>>(lv.L, lv.c, r, vis, lv.vx, lv.vz, lv.vxx, lv.vzz, lv.vxz,
                                                     lv.ratio, do_eig, ivis, rs, &ds->ratio_min); tc_note_launch();
}

// ---------------------------------------------------------------------------
// one Chebyshev step of smoother_vis with viscosityBCs fused
// ---------------------------------------------------------------------------
// v at (i, k) and its side ghosts (rows 0..b): V(-i,k)=V(i,k), V(a+i,k)=V(a-i,k)
__device__ __forceinline__ void store_with_sides(const Lay& L, double* row, int i, double v) {
    const int a = L.a;
    row[i] = v;
    if (i >= 1 && i <= SP) row[-i] = v;
    if (i >= a - SP && i <= a - 1) row[2 * a - i] = v;
}
// the top/bottom ghosts that mirror (i, k), of this column and of its side-ghost columns
__device__ __forceinline__ void store_mirror_rows(const Lay& L, double* Vout, int i, int k, double v, int RaTnz,
                                                  double visT2) {
    const int b = L.b;
    if (k >= 1 && k <= SP) store_with_sides(L, Vout + IX(L, 0, -k), i, RaTnz ? (1.0 / v / visT2) : v);
    if (k >= b - SP && k <= b - 1) store_with_sides(L, Vout + IX(L, 0, 2 * b - k), i, RaTnz ? (1.0 / v) : v);
}
__global__ void k_vis_smooth(Lay L, LevConst cc, Range2 r, const double* __restrict__ Vin, double* __restrict__ Vout,
                             const double* __restrict__ dtv, double c, const double* cdev, int RaTnz, double visT2) {
    RANGE_IK(r);
    if (!inr) return;
    if (cdev) c = *cdev;  // the factor the device-side filter loop chose
    const size_t ld = (size_t)L.ld;
    size_t x = IX(L, i, k);
    const double v0 = Vin[x], vm = Vin[x - 1], vp = Vin[x + 1], vzm = Vin[x - ld], vzp = Vin[x + ld];
    const double temp = cc.M.on ? vis_laplacian<true>(cc, i, k, v0, vm, vp, vzm, vzp)
                                : vis_laplacian<false>(cc, i, k, v0, vm, vp, vzm, vzp);
    double dts = dtv[x] * 0.99;
    double v = v0 + c * dts * temp;
    store_with_sides(L, Vout + IX(L, 0, k), i, v);
    store_mirror_rows(L, Vout, i, k, v, RaTnz, visT2);
}
void launch_vis_smooth(cudaStream_t s, const Level& lv, const double* vin, double* vout, double c, int kmin,
                       int kmax, int RaT_nonzero, double visT2, const double* cdev) {
    Range2 r{0, lv.L.a, kmin, kmax};
    k_vis_smooth<<<grid_for(r), dim3(BX, BY), 0, s>>>(lv.L, lv.c, r, vin, vout, lv.dt_vis, c, cdev, RaT_nonzero,
                                                       visT2);
    tc_note_launch();
}

// ---------------------------------------------------------------------------
// smoother_vis (smoother.f90:166-263) of a small level in one launch of a cluster: the loop
// of k_loop.cu's filter graphs, test and step in one pass with one cluster barrier.  A pass
// takes the smallest eigenvalue ratio of the current viscosity and already writes the next
// step into the other plane (the factor does not depend on the ratio); when the test then
// ends the loop that plane is dropped.  The derivative fields are written once, after the
// loop; where no test reads the ratio (interpolate) the passes only smooth.  vx null: the
// level's own viscosity (src) and derivatives stay, the result is left in A.
//
// What bounds it: the FP64 pipe, about 45 operations of 64 cycles a point and pass for 128
// points per SM at a time, and L2 latency.  The graph's loop took four nodes a step, 20 to
// 25 us whatever the level, and twelve copies around an interpolation: the viscosities of
// levels 2 to 4 of a 256x64 grid 330 + 320 + 131 us, now 116 + 65 + 35.  Larger levels keep
// the graphs: see vis_filter_fits.
// ---------------------------------------------------------------------------
#define VF_THREADS 512
#define VF_CL 16
#define VF_MAX_RATIO_METRIC 4500  // points of a stretched level with the ratio in each pass
template <bool METRIC>
__global__ void __launch_bounds__(VF_THREADS) k_vis_filter(Lay L, LevConst c, VisFltArgs q, int reset,
                                                           const double* src, double* A, double* B,
                                                           const double* __restrict__ dtv, int kmin,
                                                           int kmax, int RaTnz, double visT2, double* __restrict__ vx,
                                                           double* __restrict__ vz, double* __restrict__ vxx,
                                                           double* __restrict__ vzz, double* __restrict__ vxz,
                                                           double* __restrict__ ratio, DevScalars* ds) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank(), nt = (int)blockDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gt = rank * nt + tid, gn = C * nt;
    __shared__ unsigned long long s_warp[VF_THREADS / 32], s_all[2][VF_CL];
    const ptrdiff_t ld = (ptrdiff_t)L.ld;
    const int a = L.a, b = L.b, w = a + 1, npts = w * (kmax - kmin + 1);
    for (size_t x = gt; x < L.plane; x += gn) {
        const double v = ld_state(src + x);
        B[x] = v;
        if (A != src) A[x] = v;
    }
    // the smallest ratio of the level, from each thread's (as bits: none is negative, a NaN is never the smallest)
    auto level_min = [&](unsigned long long m, int par) {
        unsigned hi = __reduce_min_sync(0xffffffffu, (unsigned)(m >> 32));
        unsigned lo = __reduce_min_sync(0xffffffffu, (unsigned)(m >> 32) == hi ? (unsigned)m : 0xffffffffu);
        if (lane == 0) s_warp[warp] = (unsigned long long)hi << 32 | lo;
        __syncthreads();
        if (warp == 0) {
            m = lane < nt / 32 ? s_warp[lane] : ~0ull;
            hi = __reduce_min_sync(0xffffffffu, (unsigned)(m >> 32));
            lo = __reduce_min_sync(0xffffffffu, (unsigned)(m >> 32) == hi ? (unsigned)m : 0xffffffffu);
            if (lane < C) cl.map_shared_rank(&s_all[0][0], lane)[par * VF_CL + rank] = (unsigned long long)hi << 32 | lo;
        }
        cl.sync();
        m = ~0ull;
        for (int r = 0; r < C; r++) m = min(m, s_all[par][r]);
        return __longlong_as_double((long long)m);
    };
    auto point_ratio = [&](const double* V, size_t x, int i, int k, double v0, double vm, double vp, double vzm,
                           double vzp, VisDiff& d) {
        return vis_point<METRIC>(c, i, k, true, v0, vm, vp, vzm, vzp, ld_state(V + x - 1 - ld),
                                 ld_state(V + x + 1 - ld), ld_state(V + x - 1 + ld), ld_state(V + x + 1 + ld), d);
    };
    constexpr unsigned long long kInf = 0x7ffull << 52;
    // the loop's state, the same on every thread (k_vflt_init)
    int nvis = reset ? 0 : ds->vis_nvis_store, nstore = reset ? 1 : ds->vis_nn_store;
    int phase = 0, n = 0, nn = nstore, niter = q.niter0, status = 0, n_eta = 0;
    long long guard = 0;
    bool more = true, fine = false;
    auto next_outer = [&] {
        nvis += 1;
        nstore = 1;
        if (q.option == 1) {
            niter = 6;
            phase = 1;
        }
        n += 1;
        nn = 1;
        if (++guard > q.cap) {
            status = TC_ERR_LOOP_CAP;
            more = false;
        }
    };
    if (nn > niter) next_outer();
    more = true;
    cl.sync();  // both planes are the level's viscosity
    double rmin = 0.0;
    int it = 0;
    for (;; it++) {
        const double* V = (it & 1) ? B : A;
        double* W = (it & 1) ? A : B;
        const double f = phase == 0 ? __ldg(q.tabA + nn - 1) : __ldg(q.tabB + nn - 1);
        unsigned long long m = kInf;
        for (int p = gt; p < npts; p += gn) {
            const int i = p % w, k = kmin + p / w;
            const size_t x = IX(L, i, k);
            const double v0 = ld_state(V + x), vm = ld_state(V + x - 1), vp = ld_state(V + x + 1);
            const double vzm = ld_state(V + x - ld), vzp = ld_state(V + x + ld);
            const double dts = __ldg(dtv + x) * 0.99;
            const double v = v0 + f * dts * vis_laplacian<METRIC>(c, i, k, v0, vm, vp, vzm, vzp);
            store_with_sides(L, W + IX(L, 0, k), i, v);
            // (the reciprocals of rows beyond walls at RaT != 0 are not read by the passes)
            if (!RaTnz) store_mirror_rows(L, W, i, k, v, 0, visT2);
            if (!q.interpolate && i >= 1 && i <= a - 1 && k >= 1 && k <= b - 1) {
                VisDiff d;
                const double rat = point_ratio(V, x, i, k, v0, vm, vp, vzm, vzp, d);
                m = min(m, (unsigned long long)__double_as_longlong(rat));
            }
        }
        if (q.interpolate) cl.sync();
        else rmin = level_min(m, it & 1);
        // k_vflt_check
        bool stop;
        if (q.option == 1) {
            stop = (nvis >= 1 && rmin > q.eig_ratio_min) || n > 20;
            if (stop) {
                fine = true;
                n_eta = n;
            }
        } else if (q.interpolate == 0) {
            stop = rmin > q.eig_ratio;
            if (stop) nstore = nn;
        } else {
            stop = nvis >= 1;
        }
        if (stop) break;
        if (++guard > q.cap) {
            status = TC_ERR_LOOP_CAP;
            more = false;
        }
        if (++nn > niter) next_outer();
        if (!more) break;
    }
    const double* V = (it & 1) ? B : A;
    unsigned long long m = kInf;
    for (int p = gt; p < (a - 1) * (b - 1); p += gn) {
        const int i = 1 + p % (a - 1), k = 1 + p / (a - 1);
        const size_t x = IX(L, i, k);
        VisDiff d;
        const double rat = point_ratio(V, x, i, k, ld_state(V + x), ld_state(V + x - 1), ld_state(V + x + 1),
                                       ld_state(V + x - ld), ld_state(V + x + ld), d);
        if (vx != nullptr) {
            vx[x] = d.r; vz[x] = d.s; vxx[x] = d.rr; vzz[x] = d.ss; vxz[x] = d.rs;
        }
        ratio[x] = rat;
        m = min(m, (unsigned long long)__double_as_longlong(rat));
    }
    rmin = level_min(m, (it + 1) & 1);
    if (it & 1)
        for (int p = gt; p < (a + 1 + 2 * SP) * (b + 1); p += gn) {
            const size_t x = IX(L, p % (a + 1 + 2 * SP) - SP, p / (a + 1 + 2 * SP));
            A[x] = ld_state(B + x);
        }
    if (it > 0)
        for (int p = gt; p < npts; p += gn) {
            const int i = p % w, k = kmin + p / w;
            if (k <= SP || k >= b - SP) store_mirror_rows(L, A, i, k, ld_state(V + IX(L, i, k)), RaTnz, visT2);
        }
    if (gt == 0) {
        ds->ratio_min = rmin;
        ds->vis_nvis_store = nvis;
        ds->vis_nn_store = nstore;
        if (fine) {
            ds->eig_fine = rmin;
            ds->n_eta = n_eta;
        }
        if (status != 0) ds->flt_status = status;
    }
}
// The time goes with the points a thread has, the graph's hardly with the level.  A viscosity
// in one launch against the graph, spacings that are no powers of two:
//   only smoothing        one point a thread (176x44) 101 us against 209, two (224x56) 150
//                         against 204, three (272x68) 202 against 195
//   with the ratio        one (176x44) 146 against 165, two (192x48) 231 against 162
//   smoothing, stretched  one (176x44) 281 against 318, two (192x48) 495 against 317
//   ratio, stretched      some 30 divisions a point: 128x32 374 against 420, 176x44 710
//                         against 434
bool vis_filter_fits(const Level& lv, int interpolate) {
    const int a = lv.L.a, b = lv.L.b, threads = VF_THREADS * VF_CL;
    if (!interpolate && lv.c.M.on) return (a + 1) * (b + 1) <= VF_MAX_RATIO_METRIC;
    return (a + 1) * (b - 1) <= (interpolate && !lv.c.M.on ? 2 : 1) * threads;
}
// false where the device does not take the cluster: nothing ran, the loop graphs can
bool launch_vis_filter(cudaStream_t s, const Level& lv, const VisFltArgs& q, int reset, const double* src, double* A,
                       double* B, int derivatives, int kmin, int kmax, int RaT_nonzero, double visT2,
                       DevScalars* ds) {
    const int npts = (lv.L.a + 1) * (kmax - kmin + 1);
    const int nt = std::min(VF_THREADS, (npts + 128 * VF_CL - 1) / (128 * VF_CL) * 128);
    auto kernel = lv.c.M.on ? k_vis_filter<true> : k_vis_filter<false>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min(VF_CL, (npts + nt - 1) / nt), 1, 1);
    cfg.blockDim = dim3(nt, 1, 1);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cfg.gridDim.x;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (lv.no_cluster ||
        cudaLaunchKernelEx(&cfg, kernel, lv.L, lv.c, q, reset, src, A, B, (const double*)lv.dt_vis, kmin, kmax,
                           RaT_nonzero, visT2, derivatives ? lv.vx : nullptr, lv.vz, lv.vxx, lv.vzz, lv.vxz, lv.ratio,
                           ds) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    tc_note_launch();
    return true;
}

// ---------------------------------------------------------------------------
// restrict_coefficients + boundary injection of viscosityBCs_initialize
// ---------------------------------------------------------------------------
__global__ void k_restrict_vis(Lay C, Lay F, Range2 r, const double* __restrict__ vf, double* __restrict__ vc) {
    RANGE_IK(r);
    if (!inr) return;
    const int a = C.a, b = C.b;
    double v;
    if (i >= 1 && i <= a - 1 && k >= 1 && k <= b - 1) v = restrict9(vf, F, 2 * i, 2 * k);
    else if (k >= 1 && k <= b - 1) v = (i == 0) ? vf[IX(F, 0, 2 * k)] : vf[IX(F, F.a, 2 * k)];
    else v = (k == 0) ? vf[IX(F, 2 * i, 0)] : vf[IX(F, 2 * i, F.b)];
    vc[IX(C, i, k)] = v;
}
void launch_restrict_vis(cudaStream_t s, const Level& coarse, const Level& fine, const double* vfine, double* vcoarse) {
    Range2 r{0, coarse.L.a, 0, coarse.L.b};
    k_restrict_vis<<<grid_for(r), dim3(BX, BY), 0, s>>>(coarse.L, fine.L, r, vfine, vcoarse); tc_note_launch();
}

// ghosts of viscosityBCs_initialize computed from their mirror sources
__global__ void k_vis_bcs_init(Lay L, Range2 r, double* __restrict__ V, int RaTnz, double visT2) {
    RANGE_IK(r);
    if (!inr) return;
    const int a = L.a, b = L.b;
    if (i >= 0 && i <= a && k >= 0 && k <= b) return;
    int mi = (i < 0) ? -i : ((i > a) ? 2 * a - i : i);
    if (k >= 0 && k <= b) {
        V[IX(L, i, k)] = V[IX(L, mi, k)];
        return;
    }
    int mk = (k < 0) ? -k : 2 * b - k;
    double src = V[IX(L, mi, mk)];
    double g;
    if (RaTnz) g = (k < 0) ? (1.0 / src / visT2) : (1.0 / src);
    else g = src;
    V[IX(L, i, k)] = g;
}
void launch_vis_bcs_init(cudaStream_t s, const Level& coarse, double* v, int RaT_nonzero, double visT2) {
    Range2 r{-SP, coarse.L.a + SP, -SP, coarse.L.b + SP};
    k_vis_bcs_init<<<grid_for(r), dim3(BX, BY), 0, s>>>(coarse.L, r, v, RaT_nonzero, visT2); tc_note_launch();
}

// ---------------------------------------------------------------------------
// iterate_local_time_steps + folding of stream_space into 13 coefficients
// ---------------------------------------------------------------------------
__global__ void k_level_coefs(Lay L, LevConst c, Range2 r, const double* __restrict__ V, const double* __restrict__ vx,
                              const double* __restrict__ vz, const double* __restrict__ vxx,
                              const double* __restrict__ vzz, const double* __restrict__ vxz,
                              const double* __restrict__ ratio, double* __restrict__ dts, double* __restrict__ coef,
                              double* __restrict__ cA, double* __restrict__ cB, double courant_stream, int cheb,
                              MetricFold mw) {
    RANGE_IK(r);
    if (!inr) return;
    size_t x = IX(L, i, k);
    double v = V[x], ax = vx[x], az = vz[x], axx = vxx[x], azz = vzz[x], axz = vxz[x];
    if (c.M.on) {
        // stretched grid: each tap's coefficient is the operator applied to
        // that tap alone (stream_space with build = 1, iterative_solver.f90:
        // 456-561), and the local time step from the metric eigenvalues
        if (dts) {
            double eR, eI;
            eig_pair_metric(c, i, k, v, ax, az, axx, azz, axz, eR, eI);
            dts[x] = -courant_stream * 2.0 * eR / (eR * eR + eI * eI);
        }
        const int i1 = i * c.mf, k1 = k * c.mf;
        const Metric& M = c.M;
        const double x1 = mt(M.xr, i1), x2 = mt(M.xrr, i1), x3 = mt(M.xrrr, i1), x4 = mt(M.xrrrr, i1);
        const double x13 = mt(M.xr3, i1), x14 = mt(M.xr4, i1);
        const double z1 = mt(M.zs, k1), z2 = mt(M.zss, k1), z3 = mt(M.zsss, k1), z4 = mt(M.zssss, k1);
        const double z13 = mt(M.zs3, k1), z14 = mt(M.zs4, k1);
        for (int d = 0; d < TC_NCOEF; d++)
            coef[(size_t)d * L.plane + x] = stream_op_metric(mw.w[d], x1, x2, x3, x4, x13, x14, z1, z2, z3, z4, z13,
                                                             z14, v, ax, az, axx, azz, axz);
    } else {
        if (dts) {
            double eR, eI;
            eig_pair(c, v, ax, az, axx, azz, axz, eR, eI);
            dts[x] = -courant_stream * 2.0 * eR / (eR * eR + eI * eI);
        }
        double g0 = axx - azz, g1 = v, g2 = 2.0 * v, g3 = 4.0 * axz, g4 = 2.0 * ax, g5 = 2.0 * az;
#pragma unroll
        for (int d = 0; d < TC_NCOEF; d++) {
            double A = g0 * c.fold[d][0];
            A = fma(g1, c.fold[d][1], A);
            A = fma(g2, c.fold[d][2], A);
            A = fma(g3, c.fold[d][3], A);
            A = fma(g4, c.fold[d][4], A);
            A = fma(g5, c.fold[d][5], A);
            coef[(size_t)d * L.plane + x] = A;
        }
    }
    if (cheb) {
        double rr = ratio[x];
        double lb = (rr > 1.0e99) ? -2.0 : (-2.0 * (rr * rr) / (1.0 + rr * rr));
        const double la = -1.0;
        cA[x] = -lb - la;
        cB[x] = lb - la;
    }
}
void launch_level_coefs(cudaStream_t s, const Level& lv, const double* vis, int ivis, double courant_stream,
                        int cheb_level, bool with_dt) {
    (void)ivis;
    Range2 r{1, lv.L.a - 1, 1, lv.L.b - 1};
    k_level_coefs<<<grid_for(r), dim3(BX, BY), 0, s>>>(lv.L, lv.c, r, vis, lv.vx, lv.vz, lv.vxx, lv.vzz, lv.vxz,
                                                        lv.ratio, with_dt ? lv.dt_stream : nullptr, lv.coef, lv.cA,
                                                        lv.cB, courant_stream, cheb_level, lv.mfold); tc_note_launch();
}

// ---------------------------------------------------------------------------
// folded operator: RHS - L S at an interior point
// ---------------------------------------------------------------------------

// One FP64 sweep, a point per thread.  What bounds it is the FP64 pipe, 14 operations a
// point after the wait (c * dt is formed before it, ghost signs change as bits): 8.2 us a
// sweep of 1024x256 points (the pipe alone 6.1), 3.3 of 512x128; with 17 operations and the
// next launch released at the end 8.6 and 3.5.
__global__ void __launch_bounds__(256, 1) k_sweep(Lay L, Range2 r, const double* Sin, double* Sout,
                        const double* __restrict__ coef, const double* rhs,
                        const double* __restrict__ dts, const double* __restrict__ cA, const double* __restrict__ cB,
                        double c_uniform, int per_point, double temp, int Vbc) {
    RANGE_IK_DYN(r);
    const size_t x = inr ? IX(L, i, k) : 0;
    // coefficients, dt and Chebyshev denominators do not change within a solve
    double cf[TC_NCOEF], cd = 0.0;
    if (inr) {
        fold_coefs(L, coef, x, cf);
        const double c = per_point ? 2.0 / (__ldg(cA + x) + __ldg(cB + x) * temp) : c_uniform;
        cd = c * __ldg(dts + x);
    }
    pdl_entry();
    // the next sweep's blocks come in as this one's leave, their coefficients loaded meanwhile
    // (released at the end: 590 -> 572 us for 70 sweeps of 1024x256, 264 -> 241 of 200x200)
    pdl_done();
    if (!inr) return;
    double res = fold_apply(L, Sin, x, cf, ld_state(rhs + x));
    double v = fma(cd, res, ld_state(Sin + x));
    store_stream(L, Sout, i, k, v, Vbc);
}
// one point per thread: the two-point kernel (k_sweep_x2<double>, 120 registers)
// measured 18.3 against 8.5 us per level-1 sweep (half the resident warps)
static constexpr bool kSweepPairs = false;
void launch_sweep(cudaStream_t s, const Level& lv, const double* Sin, double* Sout, double c_uniform,
                  int per_point, double temp, int Vbc) {
    Range2 r{1, lv.L.a - 1, 1, lv.L.b - 1};
    if (kSweepPairs)
        launch_pdl(k_sweep_x2<double>, grid_for_shape(r, lv.sweep_bx, 2 * lv.sweep_by), dim3(lv.sweep_bx, lv.sweep_by),
                   0, s, lv.L, r, Sin, Sout, lv.coef, lv.rhs, lv.dt_stream, lv.cA, lv.cB, c_uniform, per_point, temp,
                   Vbc);
    else
        launch_pdl(k_sweep, grid_for_shape(r, lv.sweep_bx, lv.sweep_by), dim3(lv.sweep_bx, lv.sweep_by), 0, s, lv.L, r,
                   Sin, Sout, lv.coef, lv.rhs, lv.dt_stream, lv.cA, lv.cB, c_uniform, per_point, temp, Vbc);
    tc_note_launch();
}

__global__ void __launch_bounds__(256, 1) k_residual(Lay L, Range2 r, const double* S, const double* __restrict__ coef,
                           const double* rhs, double* res, RedScratch rs, double* out,
                           double div1, double div2) {
    RANGE_IK(r);
    double a = 0.0;
    double cf[TC_NCOEF];
    if (inr) fold_coefs(L, coef, IX(L, i, k), cf);
    pdl_entry();
    if (inr) {
        size_t x = IX(L, i, k);
        double v = fold_apply(L, S, x, cf, ld_state(rhs + x));
        res[x] = v;
        a = fabs(v);
    }
    reduce_to(RED_SUM, a, rs.part, rs.count, out, div1, div2);
    pdl_done();
}
void launch_residual(cudaStream_t s, const Level& lv, const double* S, RedScratch rs, double* res_out) {
    Range2 r{1, lv.L.a - 1, 1, lv.L.b - 1};
    launch_pdl(k_residual, grid_for(r), dim3(BX, BY), 0, s, lv.L, r, S, lv.coef, lv.rhs, lv.res, rs, res_out,
                                                     (double)(lv.L.a - 1), (double)(lv.L.b - 1)); tc_note_launch();
}

__global__ void k_restrict_res(Lay C, Lay F, Range2 r, const double* rf, double* rc,
                               double* zero, size_t zn) {
    pdl_entry();
    if (zero != nullptr) {
        // clear the level's correction plane in the same launch (grid-stride)
        const size_t nt = (size_t)gridDim.x * gridDim.y * blockDim.x * blockDim.y;
        const size_t t0 = ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x * blockDim.y +
                          (size_t)threadIdx.y * blockDim.x + threadIdx.x;
        for (size_t t = t0; t < zn; t += nt) zero[t] = 0.0;
    }
    RANGE_IK(r);
    if (!inr) return;
    rc[IX(C, i, k)] = restrict9(rf, F, 2 * i, 2 * k);
    pdl_done();
}
void launch_restrict_res(cudaStream_t s, const Level& coarse, const Level& fine, const double* rf, double* rhs_c,
                         double* zero) {
    Range2 r{1, coarse.L.a - 1, 1, coarse.L.b - 1};
    launch_pdl(k_restrict_res, grid_for(r), dim3(BX, BY), 0, s, coarse.L, fine.L, r, rf, rhs_c, zero,
               zero ? coarse.L.plane : (size_t)0);
    tc_note_launch();
}

// prolong (bilinear, additive) with the fine level's stream BCs fused
__global__ void k_prolong(Lay C, Lay F, Range2 r, const double* ec, double* ef, int Vbc) {
    pdl_entry();
    RANGE_IK(r);
    if (!inr) return;
    size_t x = IX(F, i, k);
    double add;
    bool ie = (i % 2) == 0, ke = (k % 2) == 0;
    if (ie && ke) add = ld_state(ec + IX(C, i / 2, k / 2));
    else if (ie) add = (ld_state(ec + IX(C, i / 2, (k - 1) / 2)) + ld_state(ec + IX(C, i / 2, (k + 1) / 2))) / 2.0;
    else if (ke) add = (ld_state(ec + IX(C, (i - 1) / 2, k / 2)) + ld_state(ec + IX(C, (i + 1) / 2, k / 2))) / 2.0;
    else
        add = (ld_state(ec + IX(C, (i - 1) / 2, (k - 1) / 2)) + ld_state(ec + IX(C, (i + 1) / 2, (k - 1) / 2)) +
               ld_state(ec + IX(C, (i + 1) / 2, (k + 1) / 2)) + ld_state(ec + IX(C, (i - 1) / 2, (k + 1) / 2))) / 4.0;
    store_stream(F, ef, i, k, ld_state(ef + x) + add, Vbc);
    pdl_done();
}
void launch_prolong(cudaStream_t s, const Level& coarse, const Level& fine, const double* ec, double* ef, int Vbc) {
    Range2 r{1, fine.L.a - 1, 1, fine.L.b - 1};
    launch_pdl(k_prolong, grid_for(r), dim3(BX, BY), 0, s, coarse.L, fine.L, r, ec, ef, Vbc); tc_note_launch();
}

// enforceBCs_stream: walls zero, ghosts mirrored from the interior
__global__ void k_stream_bcs(Lay L, Range2 r, double* __restrict__ S, int Vbc) {
    RANGE_IK(r);
    if (!inr) return;
    const int a = L.a, b = L.b;
    if (i > 0 && i < a && k > 0 && k < b) return;
    int mi = i, mk = k;
    double sg = 1.0;
    if (i < 0) { mi = -i; sg = -sg; }
    else if (i > a) { mi = 2 * a - i; sg = -sg; }
    if (k < 0) { mk = -k; if (Vbc == 0) sg = -sg; }
    else if (k > b) { mk = 2 * b - k; if (Vbc == 0) sg = -sg; }
    double v = 0.0;
    if (mi > 0 && mi < a && mk > 0 && mk < b) v = sg * S[IX(L, mi, mk)];
    S[IX(L, i, k)] = v;
}
void launch_stream_bcs(cudaStream_t s, const Level& lv, double* S, int Vbc) {
    Range2 r{-SP, lv.L.a + SP, -SP, lv.L.b + SP};
    k_stream_bcs<<<grid_for(r), dim3(BX, BY), 0, s>>>(lv.L, r, S, Vbc); tc_note_launch();
}

// ---------------------------------------------------------------------------
// coarsest grid: band assembly (Database=2 ordering), DGBEQU row scaling,
// dgbtf2 LU with partial pivoting, dgbtrs solve, scatter + BCs
// ---------------------------------------------------------------------------
// A row per thread in registers: 13 entries at most are not zero, so the equilibration
// reads no more (before, it went twice over the row's 2 kl + 1 band entries in memory: 26 us
// for 297 rows, 250 us for 10201; now 8 and 9, cold).
__global__ void k_coarse_build(Lay L, const double* __restrict__ coef, double* __restrict__ AB, double* __restrict__ rowb,
                               int n, int kl, int ku, int Vbc) {
    int pp = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (pp > n) return;
    const int nxc = L.a, nzc = L.b, N = nzc + 1, ldab = 2 * kl + ku + 1, kv1 = kl + ku + 1;
    int kp = pp - N * ((pp - 1) / N) - 1, ip = (pp - 1) / N;
    auto entry = [&](int q) { return AB + (size_t)(q - 1) * ldab + (kv1 + pp - q - 1); };  // (row pp, column q)
    const double smlnum = 2.2250738585072014e-308, bignum = 1.0 / smlnum;
    if (!(ip > 0 && ip < nxc && kp > 0 && kp < nzc)) {
        rowb[pp - 1] = 1.0;
        *entry(pp) = 1.0;
        return;
    }
    // loop order of Compute_Matrix_coarse: j=-2..2, kq ascending; taps beyond a wall mirror
    // onto the row's own column
    constexpr int od[13][3] = {{-2, 0, 3}, {-1, -1, 9}, {-1, 0, 1}, {-1, 1, 11}, {0, -2, 7}, {0, -1, 5}, {0, 0, 0},
                               {0, 1, 6},  {0, 2, 8},   {1, -1, 10}, {1, 0, 2},  {1, 1, 12}, {2, 0, 4}};
    const size_t x = IX(L, ip, kp);
    double v[13];
#pragma unroll
    for (int t = 0; t < 13; t++) v[t] = coef[(size_t)od[t][2] * L.plane + x];
    auto inside = [&](int t) {
        const int iq = ip + od[t][0], kq = kp + od[t][1];
        return iq >= 0 && iq <= nxc && kq >= 0 && kq <= nzc;
    };
#pragma unroll
    for (int t = 0; t < 13; t++)
        if (!inside(t)) v[6] = v[6] + v[t] * (od[t][0] != 0 || Vbc == 0 ? -1.0 : 1.0);
    // DGBEQU row factor of row pp (the largest entry, as integers; a NaN is never the
    // largest), then scaling of the row
    unsigned long long m = 0;
#pragma unroll
    for (int t = 0; t < 13; t++) {
        const unsigned long long k = (unsigned long long)__double_as_longlong(v[t]) & ~(1ull << 63);
        if (inside(t) && k <= (0x7ffull << 52)) m = max(m, k);
    }
    const double R = 1.0 / fmin(fmax(__longlong_as_double((long long)m), smlnum), bignum);
    rowb[pp - 1] = R;
#pragma unroll
    for (int t = 0; t < 13; t++)
        if (inside(t)) *entry(pp + N * od[t][0] + od[t][1]) = R * v[t];
}
void launch_coarse_build(cudaStream_t s, const Level& lv, double* band, double* rowb, int kl, int ku, int Vbc) {
    int n = (lv.L.a + 1) * (lv.L.b + 1);
    cudaMemsetAsync(band, 0, sizeof(double) * (size_t)(2 * kl + ku + 1) * n, s);
    k_coarse_build<<<(n + 127) / 128, 128, 0, s>>>(lv.L, lv.coef, band, rowb, n, kl, ku, Vbc); tc_note_launch();
}

// dgbtf2 on one CTA, one block barrier per column.  The columns in reach of a step
// (j..j+kl+ku) and the next few sit in a ring of column slots in shared memory.
// At step j warp 0 already works on column j+1: it applies step j to it,
// searches its pivot, swaps and scales, while the trailing warps apply step j to
// the columns behind it, a few whole columns per warp and pass (so that a row
// interchange needs no barrier), and the last warp writes column j back and loads
// the column that enters the ring.  Every element sees dgbtf2's operations in
// dgbtf2's order.
//
// What bounds it: the chain of warp 0, 0.75 to 1 us a column (update, search,
// reciprocal, scaling, barrier: FP64 latencies).  Against six barriers a column and the
// trailing update as one flat loop: 598 -> 269 us at n = 297, kl = 20 without
// interchanges, 709 -> 322 with; 1881 -> 751 us at n = 1000, kl = 8.
#define LU1_THREADS 512
#define LU1_AHEAD 4   // columns loaded ahead of the window
#define LU1_MAXKL 20  // see launch_coarse_lu; at most 31: a row per lane of warp 0
#define LU1_ROWS 2    // band rows per lane of the loading warp (2 kl + ku + 1 <= 64)
__global__ void __launch_bounds__(LU1_THREADS) k_coarse_lu(double* __restrict__ ABg, int* __restrict__ ipiv, int n,
                                                           int kl, int ku, int* info_out) {
    extern __shared__ double sm[];
    const int ldab = 2 * kl + ku + 1, KV = ku + kl, C = KV + 1 + LU1_AHEAD;
    __shared__ double mult[2][LU1_MAXKL + 1];
    __shared__ int sCode[2];  // pivot row offset * 2 + (pivot != 0), per step parity
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = LU1_THREADS / 32;
    // column cl (1-based) as an array of band rows 1..ldab; at = j % C
    int at_j = 0;
    auto col = [&](int cl) { return sm + (size_t)(cl % C) * ldab - 1; };
    auto col_after = [&](int c) {  // column j + c, 0 <= c <= KV
        int q = at_j + c;
        if (q >= C) q -= C;
        return sm + q * ldab - 1;
    };
    auto nonzero = [](double x) { return (unsigned long long)(__double_as_longlong(x) << 1) != 0ull; };
    // loads column cl with dgbtf2's zeroed fill-in rows
    auto load_col = [&](int cl, int t0, int nt) {
        double* d = col(cl);
        const double* g = ABg + (size_t)(cl - 1) * ldab - 1;
        const int z0 = (cl > KV) ? 1 : KV - cl + 2;  // rows z0..kl of the columns ku+2.. are fill-in
        for (int t = 1 + t0; t <= ldab; t += nt) d[t] = (cl >= ku + 2 && t >= z0 && t <= kl) ? 0.0 : g[t];
    };
    for (int cl = 1 + warp; cl <= min(n, KV + LU1_AHEAD); cl += NW) load_col(cl, lane, 32);
    double pf[LU1_ROWS];  // the loader's next column, loaded a step before it is stored
    int pf_col = 0;
    __syncthreads();
    int JU = 1, info = 0;
    const int G = max(1, 64 / kl);  // columns of a trailing warp's pass
    int code = 0;
    for (int j = 0; j <= n; j++) {
        // step j (j = 0: none) is prepared: pivot code, multipliers, column j
        const int KM = min(kl, n - j), JP = code >> 1;
        const bool nz = j > 0 && (code & 1) != 0;
        const double* mj = mult[j & 1];
        if (j > 0) {
            if (nz) JU = max(JU, min(j + ku + JP - 1, n));
            else if (info == 0) info = j;
        }
        if (warp == 0) {
            if (j + 1 <= n) {
                // column j+1: rows t = 0..KM1 below and on its diagonal, two per lane
                const int KM1 = min(kl, n - j - 1);
                double* a = col_after(1) + KV + 1;
                double v = lane <= KM1 ? a[lane] : 0.0;
                if (nz && j + 1 <= JU) {
                    const double oldtop = a[-1], top = a[JP - 2];
                    const double temp = -top;
                    if (lane + 1 == JP - 1) v = oldtop;  // lane: row lane + 1 of step j
                    if (lane < KM && nonzero(temp)) v = v + mj[lane + 1] * temp;
                    __syncwarp();
                    if (lane == 0 && JP != 1) a[-1] = top;
                }
                // idamax: the first row of the largest |value| (as integers; a NaN is never the largest)
                unsigned long long key = (unsigned long long)__double_as_longlong(v) & ~(1ull << 63);
                key = (key > (0x7ffull << 52) || lane > KM1) ? 0 : key + 1;
                const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
                const bool tops = (unsigned)(key >> 32) == hi;
                const unsigned lo = __reduce_max_sync(0xffffffffu, tops ? (unsigned)key : 0u);
                const int bi = __ffs(__ballot_sync(0xffffffffu, tops && (unsigned)key == lo)) - 1;
                const double piv = __shfl_sync(0xffffffffu, v, bi);
                const double first = __shfl_sync(0xffffffffu, v, 0);
                const int nzp = nonzero(piv) ? 1 : 0;
                if (nzp) {
                    const double rcp = 1.0 / piv;
                    if (lane == bi) v = first;
                    v = lane == 0 ? piv : rcp * v;
                }
                if (lane <= KM1) {
                    a[lane] = v;
                    mult[(j + 1) & 1][lane] = v;
                }
                if (lane == 0) {
                    sCode[(j + 1) & 1] = (bi + 1) * 2 + nzp;
                    ipiv[j] = bi + j + 1;
                }
            }
        } else if (warp == NW - 1) {
            if (j > 0) {
                const double* d = col_after(0);
                double* g = ABg + (size_t)(j - 1) * ldab - 1;
                for (int t = 1 + lane; t <= ldab; t += 32) g[t] = d[t];
            }
            // column j+KV+AHEAD-1 takes the slot of column j-2, written back two
            // steps ago (at j = 2 a slot that was never used)
            if (pf_col > 0) {
                double* e = col(pf_col);
#pragma unroll
                for (int u = 0; u < LU1_ROWS; u++) {
                    const int t = 1 + lane + 32 * u;
                    if (t <= ldab) e[t] = pf[u];
                }
            }
            pf_col = (j >= 1 && j + KV + LU1_AHEAD <= n) ? j + KV + LU1_AHEAD : 0;
            if (pf_col > 0) {
                const double* g = ABg + (size_t)(pf_col - 1) * ldab - 1;
#pragma unroll
                for (int u = 0; u < LU1_ROWS; u++) {
                    const int t = 1 + lane + 32 * u;
                    pf[u] = (t <= ldab && t > kl) ? g[t] : 0.0;  // rows 1..kl: fill-in
                }
            }
        } else if (nz) {
            // columns j+2..JU, G at a time: at most 64 elements, two per lane
            for (int c0 = 2 + (warp - 1) * G; c0 <= JU - j; c0 += (NW - 2) * G) {
                double v[2], top[2];
                double *at[2], *topat[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int e = lane + 32 * u;
                    at[u] = topat[u] = nullptr;
                    int q = (e >= KM) + (e >= 2 * KM) + (e >= 3 * KM);
                    if (G > 4) q = e / KM;
                    const int c = c0 + q, t = 1 + e - q * KM;
                    if (e >= G * KM || c > JU - j) continue;
                    double* a = col_after(c) + KV + 1 - c;  // row j of column j + c
                    top[u] = a[JP - 1];
                    const double temp = -top[u];
                    v[u] = (t == JP - 1) ? a[0] : a[t];
                    if (nonzero(temp)) v[u] = v[u] + mj[t] * temp;
                    at[u] = a + t;
                    if (t == 1 && JP != 1) topat[u] = a;
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (at[u] != nullptr) *at[u] = v[u];
                    if (topat[u] != nullptr) *topat[u] = top[u];
                }
                __syncwarp();
            }
        }
        __syncthreads();
        if (++at_j == C) at_j = 0;
        if (j < n) code = sCode[(j + 1) & 1];
    }
    if (tid == 0) *info_out = info;
}
// dgbtf2 on one CTA with the band in global memory: bands too wide for the kernels
// above and below (kl > 480).
__global__ void k_coarse_lu_global(double* __restrict__ AB, int* __restrict__ ipiv, int n, int kl, int ku,
                                   int* info_out) {
    const int ldab = 2 * kl + ku + 1, KV = ku + kl;
    const int tid = threadIdx.x, nth = blockDim.x;
    __shared__ int sJP, sJU, sInfo;
    __shared__ double sPiv;
    if (tid == 0) { sJU = 1; sInfo = 0; }
    __syncthreads();
#define A_(rw, cl) AB[(size_t)((rw) - 1) + (size_t)((cl) - 1) * ldab]
    for (int j = ku + 2; j <= min(KV, n); j++)
        for (int i = KV - j + 2 + tid; i <= kl; i += nth) A_(i, j) = 0.0;
    __syncthreads();
    for (int j = 1; j <= n; j++) {
        if (j + KV <= n)
            for (int i = 1 + tid; i <= kl; i += nth) A_(i, j + KV) = 0.0;
        const int KM = min(kl, n - j);
        __syncthreads();
        if (tid < 32) {
            // idamax: first index of the largest |value| among rows KV+1..KV+1+KM
            double best = -1.0;
            int bi = 1 << 30;
            for (int t = 1 + tid; t <= KM + 1; t += 32) {
                double v = fabs(A_(KV + t, j));
                if (v > best) { best = v; bi = t; }
            }
            for (int off = 16; off > 0; off >>= 1) {
                double ob = __shfl_down_sync(0xffffffffu, best, off);
                int oi = __shfl_down_sync(0xffffffffu, bi, off);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            if (tid == 0) {
                sJP = bi;
                ipiv[j - 1] = bi + j - 1;
                sPiv = A_(KV + bi, j);
                if (sPiv != 0.0) sJU = max(sJU, min(j + ku + bi - 1, n));
                else if (sInfo == 0) sInfo = j;
            }
        }
        __syncthreads();
        const int JP = sJP, JU = sJU;
        if (sPiv != 0.0) {
            if (JP != 1) {
                for (int c = tid; c <= JU - j; c += nth) {
                    double t0 = A_(KV + JP - c, j + c);
                    A_(KV + JP - c, j + c) = A_(KV + 1 - c, j + c);
                    A_(KV + 1 - c, j + c) = t0;
                }
                __syncthreads();
            }
            if (KM > 0) {
                const double rcp = 1.0 / A_(KV + 1, j);
                for (int t = 1 + tid; t <= KM; t += nth) A_(KV + 1 + t, j) = rcp * A_(KV + 1 + t, j);
                __syncthreads();
                const int ncol = JU - j;
                for (int e = tid; e < ncol * KM; e += nth) {
                    int c = 1 + e / KM, t = 1 + e % KM;
                    double temp = -A_(KV + 1 - c, j + c);
                    if (temp != 0.0) A_(KV + 1 + t - c, j + c) = A_(KV + 1 + t - c, j + c) + A_(KV + 1 + t, j) * temp;
                }
            }
        }
        __syncthreads();
    }
#undef A_
    if (tid == 0) *info_out = sInfo;
}
// The same factorisation with a panel of LUP_NB columns per launch, for wider bands.
// Launch p factors panel p and applies panel p-1 to the columns behind it, so that
// only the panel's own chain of pivots is serial:
//  - Cluster 0 takes one column of the panel per CTA, one row per thread.  Each CTA
//    applies each step of the panel as it arrives, then searches its pivot.  While one
//    warp does that and divides, the others send the unscaled column to the cluster's
//    CTAs (st.async); the pivot and its reciprocal follow, and the receivers scale.
//    The second half of its threads brings a column of panel p+1 up to date in the
//    same way, with the steps of panel p-1 first.
//  - The other CTAs apply the steps of panel p-1 to one column per warp, in registers.
// A column sees the steps before it in order, each as interchange and update with a
// separate multiply and add: dgbtf2's operations in dgbtf2's order.  The fill-in rows
// of the band are zero on entry (launch_coarse_build clears the band).
//
// What bounds it: the chain of pivots, 2400 cycles a column at kl = 202 (1800 at 20):
// update 750 (three dependent FP64 operations on seven warps, the pipe does 2 lanes a
// cycle), search 600, reciprocal 620, message 400.  Everything else is kept off it.
// Before, one cluster of 8 CTAs with the whole window in its shared memory, every
// column's update on the chain: n = 10201, kl = 202 (a 200x200 grid halved once) 73 ms,
// now 12.7; one CTA for n = 400, kl = 63: 2.36 ms, now 0.46.
#define LUP_NB 16
#define LUP_CL 16              // CTAs of the panel's cluster: one per column
#define LUP_WAIT (1 << 20)     // polls of a wait for a column's multipliers
#define LUP_TEST_WAIT (1 << 14)  // polls of the timeout-path test's word
template <int T>
__global__ void __launch_bounds__(2 * T) k_lu_panel(double* ABg, int* ipiv, int n, int kl, int ku, int p, DevScalars* ds,
                                                    const int* test_flag) {
    constexpr int NB = LUP_NB, NW = T / 32, R = T / 32;  // NW: warps of a column
    extern __shared__ __align__(16) double smd[];  // [2][NB][T]: multipliers of panel p-1, unscaled columns of this one
    double* msg = smd + NB * T;
    __shared__ __align__(8) unsigned long long bar[NB];
    __shared__ __align__(16) unsigned long long head[NB][2];  // per column of the panel: code, reciprocal
    __shared__ int s_ju[NB], s_op[NB], s_max;
    __shared__ __align__(16) double s_cols[2][2][T];
    __shared__ double s_rcp, s_val[2][NW];
    __shared__ unsigned long long s_key[2][NW];
    __shared__ int s_idx[2][NW], s_bi;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldab = 2 * kl + ku + 1, KV = kl + ku;
    const int j0 = p * NB + 1, b0 = j0 - NB;  // first column (1-based); row of offset 0
    const bool panel = blockIdx.x < LUP_CL;
    const int c = blockIdx.x;                 // the panel's column of this CTA
    const int last = min(LUP_CL, n - j0 + 1) - 1;
    auto at = [&](int r, int q) { return ABg + (size_t)(q - 1) * ldab + (KV + r - q); };
    auto nonzero = [](double x) { return (unsigned long long)(__double_as_longlong(x) << 1) != 0ull; };
    // the first lane with the largest key
    auto first_max = [](unsigned long long key) {
        const unsigned hi = (unsigned)(key >> 32), top = __reduce_max_sync(0xffffffffu, hi);
        unsigned who = __ballot_sync(0xffffffffu, hi == top);
        if (__popc(who) > 1) {
            const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)key : 0u);
            who = __ballot_sync(0xffffffffu, hi == top && (unsigned)key == lo);
        }
        return __ffs(who) - 1;
    };
    // rows sent of column i: its pivot rows, in 16-byte pairs
    auto sent_from = [&](int i) { return (NB + i) & ~1; };
    auto sent_bytes = [&](int i) { return 8 * (((NB + i + min(kl, n - j0 - i)) | 1) + 1 - sent_from(i)); };
    if (panel) {
        if (tid < NB) mbar_init(smem_addr(&bar[tid]), 1);
        __syncthreads();
        if (tid <= last) mbar_arrive_expect(smem_addr(&bar[tid]), sent_bytes(tid) + 16);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        cluster_arrive();
    }
    pdl_entry();
    pdl_done();
    if (tid == 0) s_max = 0;
    __syncthreads();
    if (p > 0 && tid < NB) {
        const int ju = ld_state(&ds->lu_ju[(p - 1) & 1][tid]);
        s_ju[tid] = ju;
        s_op[tid] = ld_state(ipiv + b0 - 1 + tid) - b0;
        atomicMax(&s_max, ju);
    }
    if (panel) {
        // threads 0..T-1: column c of the panel; T..2T-1: column c of the next panel,
        // which follows the steps at its own pace
        const bool ahead = tid >= T;
        const int o = tid & (T - 1), jc = j0 + c + (ahead ? NB : 0), r = b0 + o;
        const bool live = c <= last, valid = jc <= n && r >= max(1, jc - KV) && r <= min(n, jc + kl);
        double v = valid ? ld_state(at(r, jc)) : 0.0;
        double(*s_cur)[T] = s_cols[ahead ? 1 : 0];
        // the column as its other threads see it: s_cur[x]
        int x = 0;
        auto publish = [&] {
            x ^= 1;
            s_cur[x][o] = v;
            asm volatile("bar.sync %0, %1;" ::"r"(ahead ? 2 : 1), "n"(T) : "memory");
        };
        // step k (offset ok, pivot offset op) on this column: interchange and update
        auto step = [&](bool on, int ok, int op, auto mult) {
            const double top = s_cur[x][op], old = s_cur[x][ok], temp = -top;
            if (on) {
                if (o == op) v = old;
                if (o == ok) v = top;
                if (nonzero(temp) && o > ok && o <= ok + kl && r <= n) v = v + mult() * temp;
            }
        };
        __syncthreads();
        publish();
        bool dead = false;
        if (test_flag != nullptr) {
            if (o == 0)
                for (int it = 0; *(volatile const int*)test_flag == 0 && it < LUP_TEST_WAIT; it++) {
                }
            dead = true;
        }
        // the step of column i of this panel, once it is here; its JU and info.  Every thread passes the
        // same barriers, also if a wait gave up (it then takes no step and keeps its JU and info)
        auto arrived = [&](int i, int& ju, int& info) {
            int it = 0;
            bool here;
            while (!(here = mbar_try_wait(smem_addr(&bar[i]), 0)))
                if (dead || ++it > LUP_WAIT) { dead = true; break; }
            const unsigned long long code = here ? head[i][0] : (unsigned long long)info << 36 | (unsigned long long)ju << 12;
            const double rcp = __longlong_as_double((long long)head[i][1]);
            const int ok = NB + i, op = (int)(code >> 1) & (T - 1);
            ju = (int)(code >> 12) & 0xffffff;
            info = (int)(code >> 36);
            step((code & 1) && jc <= ju, ok, op, [&] { return rcp * msg[i * T + (o == op ? ok : o)]; });
        };
        // The end of a panel's CTA: no CTA leaves while another still reads or writes its
        // shared memory.  A thread that gave up reports it and waits, within the same bound,
        // for the columns still on their way here, before the barrier and, when all are sent, after it.
        auto leave = [&] {
            auto landed = [&] {
                for (int i = 0; dead && live && i <= last; i++)
                    for (int it = 0; it < LUP_WAIT && !mbar_try_wait(smem_addr(&bar[i]), 0); it++) {
                    }
            };
            if (dead) atomicExch(&ds->visit_timeout, 1);
            landed();
            __syncwarp();
            cluster_arrive_relaxed();
            cluster_wait();
            landed();
        };
        if (ahead) {
            // The FP64 pipe is the panel's while this CTA holds the pivot chain: these
            // columns wait until it has passed -- at once, with the steps of panel p-1
            // done, or just before it comes, by the time they have until then.  (n = 1089,
            // kl = 62: 1.21 ms; all at once 1.72; the lines at 3 and 8 instead of 6 and 10 1.22,
            // at 9 and 12 1.27.  kl = 202: 3.17, 4.89, 3.26, 3.67; kl = 300: 3.14, 4.51, 3.23, 3.55)
            auto chain_passed = [] { asm volatile("bar.sync 3, %0;" ::"n"(2 * T) : "memory"); };
            const int pause = c < 6 ? -1 : c < 10 ? 0 : c - 1;
            int ju = 0, info = 0;
            if (live && pause < 0) chain_passed();
            if (p > 0) {
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    const int k = b0 + i;
                    smd[i * T + o] = (r > k && r <= min(n, k + kl)) ? ld_state(at(r, k)) : 0.0;
                }
#pragma unroll 1
                for (int i = 0; i < NB; i++) {
                    step(jc <= s_ju[i], i, s_op[i], [&] { return smd[i * T + o]; });
                    publish();
                }
            }
            cluster_wait();  // every mbarrier of the cluster is set up
#pragma unroll 1
            for (int i = 0; live && i <= last; i++) {
                if (i == pause) chain_passed();
                arrived(i, ju, info);
                publish();
            }
            if (valid) *at(r, jc) = v;
            leave();
            return;
        }
        cluster_wait();
        int ju = 1, info = 0;
        if (c == 0 && p > 0) {
            ju = ld_state(&ds->lu_run);
            info = ld_state(&ds->lu_info);
        }
        // the unscaled column to CTA c + 1 + l (modulo the columns of the panel)
        auto send_column = [&](int l) {
            const int q = c + 1 + l <= last ? c + 1 + l : c + l - last, t = sent_from(c);
            bulk_to_cluster(cluster_addr(smem_addr(msg + c * T + t), q), smem_addr(&s_cur[x][t]), sent_bytes(c),
                            cluster_addr(smem_addr(&bar[c]), q));
        };
        if (live) {
            // The search and the division also run once before the first step: that brings
            // their code into the instruction cache before the chain waits for it.
            const int ok = NB + c, KM = min(kl, n - jc);
#pragma unroll 1
            for (int i = 0; i <= c; i++) {
                if (i > 0) arrived(i - 1, ju, info);
                if (i > 0 && i < c) {
                    publish();
                    continue;
                }
                // idamax (as integers; a NaN is never the largest)
                unsigned long long key = (unsigned long long)__double_as_longlong(v) & ~(1ull << 63);
                key = (key > (0x7ffull << 52) || o < ok || o > ok + KM) ? 0 : key + 1;
                if (lane == first_max(key)) {
                    s_key[x][warp] = key;
                    s_idx[x][warp] = o;
                    s_val[x][warp] = v;
                }
                const bool own = i == c;
                if (own && o >= sent_from(c) && 8 * (o - sent_from(c)) < sent_bytes(c))
                    st_async8(cluster_addr(smem_addr(msg + c * T + o), c < last ? c + 1 : 0),
                              (unsigned long long)__double_as_longlong(v),
                              cluster_addr(smem_addr(&bar[c]), c < last ? c + 1 : 0));
                publish();
                if (warp == 0) {
                    key = lane < NW ? s_key[x ^ 1][lane] : 0;
                    int op = lane < NW ? s_idx[x ^ 1][lane] : 0;
                    double piv = lane < NW ? s_val[x ^ 1][lane] : 0.0;
                    const int w = first_max(key);
                    key = __shfl_sync(0xffffffffu, key, w);
                    op = __shfl_sync(0xffffffffu, op, w);
                    piv = __shfl_sync(0xffffffffu, piv, w);
                    if (key == 0) {  // no number among them
                        op = ok;
                        piv = s_cur[x][ok];
                    }
                    const bool nz = nonzero(piv);
                    double rcp = 0.0;
                    if (nz) rcp = 1.0 / piv;
                    if (own) {
                        if (nz) ju = max(ju, min(b0 + op + ku, n));
                        else if (info == 0) info = jc;
                    }
                    const unsigned long long code = (unsigned long long)info << 36 | (unsigned long long)ju << 12 |
                                                    (unsigned long long)op << 1 | (nz ? 1 : 0);
                    // to every CTA, the next one first
                    if (own && lane <= last) {
                        const int q = c + 1 + lane <= last ? c + 1 + lane : c + lane - last;
                        st_async16(cluster_addr(smem_addr(head[c]), q), code,
                                   (unsigned long long)__double_as_longlong(rcp), cluster_addr(smem_addr(&bar[c]), q));
                    }
                    if (lane == 0) {
                        s_bi = op;
                        s_rcp = rcp;
                    }
                }
            }
            asm volatile("bar.arrive 3, %0;" ::"n"(2 * T) : "memory");
            fence_async();
            asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
            if (tid >= 1 && tid <= last) send_column(tid);
            const int op = s_bi;
            const double piv = s_cur[x][op];
            if (nonzero(piv)) {
                if (o == op) v = s_cur[x][ok];
                if (o == ok) v = piv;
                if (o > ok && o <= ok + KM) v = s_rcp * v;
            }
            if (valid) *at(r, jc) = v;
            if (tid == 0) {
                ipiv[jc - 1] = b0 + op;
                ds->lu_ju[p & 1][c] = nonzero(piv) ? ju : 0;
                if (c == last) {
                    ds->lu_run = ju;
                    ds->lu_info = info;
                }
            }
        }
        leave();
        return;
    }
    // columns behind these two panels: steps of panel p-1
    if (tid < T) {
        const int r = b0 + tid;
#pragma unroll 4
        for (int i = 0; i < NB; i++) {
            const int k = b0 + i;
            smd[i * T + tid] = (r > k && r <= min(n, k + kl)) ? ld_state(at(r, k)) : 0.0;
        }
    }
    __syncthreads();
    const int nct = gridDim.x - LUP_CL, reach = s_max;
    for (int q = j0 + 2 * NB + (int)(blockIdx.x - LUP_CL) + warp * nct; q <= reach; q += nct * 2 * NW) {
        const int rlo = max(1, q - KV), rhi = min(n, min(q + kl, b0 + NB - 1 + kl));
        double v[R];
#pragma unroll
        for (int u = 0; u < R; u++) {
            const int r = b0 + lane + 32 * u;
            v[u] = (r >= rlo && r <= rhi) ? ld_state(at(r, q)) : 0.0;
        }
#pragma unroll 1
        for (int i = 0; i < NB; i++) {
            if (q > s_ju[i]) continue;
            const int op = s_op[i], up = op >> 5, KM = min(kl, n - (b0 + i));
            double x = v[0];
#pragma unroll
            for (int u = 1; u < R; u++)
                if (u == up) x = v[u];
            const double top = __shfl_sync(0xffffffffu, x, op & 31), old = __shfl_sync(0xffffffffu, v[0], i);
            const double temp = -top;
            if (lane == (op & 31)) {
#pragma unroll
                for (int u = 0; u < R; u++)
                    if (u == up) v[u] = old;
            }
            if (lane == i) v[0] = top;
            if (nonzero(temp)) {
#pragma unroll
                for (int u = 0; u < R; u++) {
                    const int o = lane + 32 * u;
                    if (o > i && o <= i + KM) v[u] = v[u] + smd[i * T + o] * temp;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < R; u++) {
            const int r = b0 + lane + 32 * u;
            if (r >= rlo && r <= rhi) *at(r, q) = v[u];
        }
    }
}
// false where the device does not take a cluster of LUP_CL such CTAs (nothing ran); a launch
// refused later leaves its error for the solve's next read
template <int T>
bool launch_lu_panels(cudaStream_t s, double* band, int* ipiv, int n, int kl, int ku, DevScalars* ds,
                      const int* test_flag) {
    const size_t smem = sizeof(double) * 2 * LUP_NB * T;
    cudaFuncSetAttribute(k_lu_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_lu_panel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    // the columns behind the panel two to four per SM, on up to seven clusters with the
    // panel's: an eighth of the chip stays free for the next launch's panel, whose CTAs then
    // share no SM with this launch's (n = 2600, kl = 202: 3.17 ms; with eight clusters 3.47,
    // with six 3.38; n = 1800, kl = 300: 3.14, 5.48 and 3.31; the same below kl = 126)
    const int clusters = 1 + std::min(6, (kl + ku + 31) / 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(LUP_CL * clusters, 1, 1);
    cfg.blockDim = dim3(2 * T, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = LUP_CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    static PerDevice fits;
    if (fits.get([&] {
            int c = 0;
            if (cudaOccupancyMaxActiveClusters(&c, k_lu_panel<T>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
            return c;
        }) < 1)
        return false;
    cfg.numAttrs = 2;
    for (int p = 0; p * LUP_NB < n; p++) {
        if (p == 0) cfg.gridDim.x = LUP_CL;
        else cfg.gridDim.x = LUP_CL * clusters;
        if (cudaLaunchKernelEx(&cfg, k_lu_panel<T>, band, ipiv, n, kl, ku, p, ds, test_flag) != cudaSuccess) {
            if (p == 0) cudaGetLastError();
            return p != 0;
        }
        tc_note_launch();
    }
    return true;
}

void launch_coarse_lu(cudaStream_t s, const Level& lv, double* band, int* ipiv, int n, int kl, int ku, DevScalars* ds,
                      const int* test_flag) {
    const int ldab = 2 * kl + ku + 1;
    const size_t ring = sizeof(double) * (size_t)ldab * (kl + ku + 1 + LU1_AHEAD);
    // one CTA for the narrowest bands: no messages and no launches between the columns
    // (n = 1000, kl = 8: 751 us against 1033 by panels), while its FP64 pipe keeps up with
    // the chain of pivots (n = 552, kl = 24: 938 against 575)
    if (kl <= LU1_MAXKL && ldab <= 32 * LU1_ROWS && ring <= 48 * 1024) {
        k_coarse_lu<<<1, LU1_THREADS, ring, s>>>(band, ipiv, n, kl, ku, &ds->lu_info); tc_note_launch();
        return;
    }
    // one row per thread: the rows that two panels' steps reach
    const int rows = kl + 2 * LUP_NB;
    if (lv.no_cluster) {
    } else if (rows <= 64 ? launch_lu_panels<64>(s, band, ipiv, n, kl, ku, ds, test_flag)
        : rows <= 128 ? launch_lu_panels<128>(s, band, ipiv, n, kl, ku, ds, test_flag)
        : rows <= 256 ? launch_lu_panels<256>(s, band, ipiv, n, kl, ku, ds, test_flag)
        : rows <= 512 && launch_lu_panels<512>(s, band, ipiv, n, kl, ku, ds, test_flag)) return;
    k_coarse_lu_global<<<1, 512, 0, s>>>(band, ipiv, n, kl, ku, &ds->lu_info); tc_note_launch();
}

// RN(x / d) from y + y2 = 1 / d to twice the precision: a quotient within one ulp, and
// Markstein's correction with its exact remainder (IBM J. Res. Dev. 34, 1990).  y = 0: d
// is near the ends of the range.
__device__ __forceinline__ double solve_quot(double x, double d, double y, double y2) {
    const double q0 = fma(x, y, x * y2);
    double q = fma(fma(-q0, d, x), y, q0);
    const unsigned hi = (unsigned)__double2hiint(x);
    if ((hi >> 20 & 0x7ff) - 600u > 846u || __double2hiint(y) == 0) {
        if (((hi << 1) | (unsigned)__double2loint(x)) != 0) q = x / d;  // 0 where x is
    }
    return q;
}
__device__ __forceinline__ void solve_recip(double d, double& y, double& y2) {
    const unsigned ed = (unsigned)__double2hiint(d) >> 20 & 0x7ff;
    y = ed - 600u > 846u ? 0.0 : 1.0 / d;
    y2 = fma(-y, d, 1.0) * y;
}

// Explicit inverse of the factored coarse matrix: column j of A^-1 is the
// DGBTRS solve (row interchanges + L solve, then dtbsv) of the unit vector
// e_j.  One warp per column, the vector in shared memory.  Stored row-major
// (Ainv[p*n + q]) for the coalesced products below.
//
// What bounds it: the chain of FP64 operations of a column, 64 cycles each, so each
// warp has a scheduler of its own (four per CTA) and the pivots' reciprocals, formed
// once, replace most of each division.  The band comes from L1/L2, FW rows per lane below
// the diagonal and 2 FW above, loaded four steps ahead.  286 -> 180 us at n = 297,
// kl = 20 (before: eight warps per CTA, divisions, the band staged in shared memory where
// it fits); n = 289, kl = 34: 346 us without the loads ahead, 239 with them.
#define CI_WARPS 4
template <int FW>
__global__ void __launch_bounds__(32 * CI_WARPS) k_coarse_inverse(const double* __restrict__ ABg,
                                                                  const int* __restrict__ ipiv, int n, int kl, int ku,
                                                                  double* __restrict__ Ainv) {
    constexpr int D = 4;  // steps loaded ahead
    extern __shared__ double sm[];
    const int ldab = 2 * kl + ku + 1, KD = ku + kl + 1, K = kl + ku;
    const int tid = threadIdx.x, nth = 32 * CI_WARPS, lane = tid & 31, warp = tid >> 5;
    double *sd = sm, *sy = sd + n, *sy2 = sy + n, *Bw = sy2 + n + (size_t)warp * n;
#define A_(rw, cl) ABg[(size_t)((rw) - 1) + (size_t)((cl) - 1) * ldab]
    for (int t = tid; t < n; t += nth) {
        sd[t] = __ldg(&A_(K + 1, t + 1));
        solve_recip(sd[t], sy[t], sy2[t]);
    }
    __syncthreads();
    const int j = blockIdx.x * CI_WARPS + warp + 1;  // column of A^-1 (1-based)
    if (j > n) return;
    auto nonzero = [](double x) { return (unsigned long long)(__double_as_longlong(x) << 1) != 0ull; };
    for (int t = lane; t < n; t += 32) Bw[t] = (t == j - 1) ? 1.0 : 0.0;
    __syncwarp();
    {
        double f[D][FW];
        int pv[D];
        auto fetch = [&](int jj, int q) {
            if (jj > n - 1) return;
            pv[q] = __ldg(ipiv + jj - 1);
#pragma unroll
            for (int u = 0; u < FW; u++) {
                const int t = 1 + lane + 32 * u;
                f[q][u] = t <= min(kl, n - jj) ? __ldg(&A_(KD + t, jj)) : 0.0;
            }
        };
        const int first = max(1, j - kl);  // earlier steps interchange and add zeros
#pragma unroll
        for (int q = 0; q < D; q++) fetch(first + q, q);
        for (int j0 = first; j0 <= n - 1; j0 += D) {
#pragma unroll
            for (int q = 0; q < D; q++) {
                const int jj = j0 + q;
                if (jj > n - 1) break;
                const int LM = min(kl, n - jj), Lr = pv[q];
                const double top = Bw[Lr - 1];
                if (Lr != jj) {
                    __syncwarp();
                    if (lane == 0) { Bw[Lr - 1] = Bw[jj - 1]; Bw[jj - 1] = top; }
                    __syncwarp();
                }
                const double temp = -top;
                if (nonzero(temp)) {
#pragma unroll
                    for (int u = 0; u < FW; u++) {
                        const int t = 1 + lane + 32 * u;
                        if (t <= LM) Bw[jj + t - 1] = Bw[jj + t - 1] + f[q][u] * temp;
                    }
                    for (int t = 1 + lane + 32 * FW; t <= LM; t += 32)
                        Bw[jj + t - 1] = Bw[jj + t - 1] + __ldg(&A_(KD + t, jj)) * temp;
                }
                __syncwarp();
                fetch(jj + D, q);
            }
        }
    }
    double g[D][2 * FW];
    auto fetch = [&](int jj, int q) {
        if (jj < 1) return;
#pragma unroll
        for (int u = 0; u < 2 * FW; u++) {
            const int i = jj - 1 - lane - 32 * u;
            g[q][u] = i >= max(1, jj - K) ? __ldg(&A_(K + 1 - jj + i, jj)) : 0.0;
        }
    };
#pragma unroll
    for (int q = 0; q < D; q++) fetch(n - q, q);
    for (int j0 = n; j0 >= 1; j0 -= D) {
#pragma unroll
        for (int q = 0; q < D; q++) {
            const int jj = j0 - q;
            if (jj < 1) break;
            const double bj = Bw[jj - 1];
            if (nonzero(bj)) {
                const double temp = solve_quot(bj, sd[jj - 1], sy[jj - 1], sy2[jj - 1]);
                __syncwarp();
                if (lane == 0) Bw[jj - 1] = temp;
#pragma unroll
                for (int u = 0; u < 2 * FW; u++) {
                    const int i = jj - 1 - lane - 32 * u;
                    if (i >= max(1, jj - K)) Bw[i - 1] = Bw[i - 1] - temp * g[q][u];
                }
                for (int i = jj - 1 - lane - 64 * FW; i >= max(1, jj - K); i -= 32)
                    Bw[i - 1] = Bw[i - 1] - temp * __ldg(&A_(K + 1 - jj + i, jj));
            }
            __syncwarp();
            fetch(jj - D, q);
        }
    }
#undef A_
    for (int p = lane; p < n; p += 32) Ainv[(size_t)p * n + (j - 1)] = Bw[p];
}
void launch_coarse_inverse(cudaStream_t s, const double* band, const int* ipiv, int n, int kl, int ku, double* Ainv) {
    const size_t sm = sizeof(double) * (3 + CI_WARPS) * (size_t)n;
    auto go = [&](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        kernel<<<(n + CI_WARPS - 1) / CI_WARPS, 32 * CI_WARPS, sm, s>>>(band, ipiv, n, kl, ku, Ainv); tc_note_launch();
    };
    if (kl <= 32) go(k_coarse_inverse<1>);
    else if (kl <= 64) go(k_coarse_inverse<2>);
    else go(k_coarse_inverse<4>);
}

// Coarsest-level solve as x = A^-1 (RowB .* RHS) (Compute_coarse_vector,
// DGBTRS, Stream_grid_coarse): one warp per interior unknown (the boundary
// unknowns are zero: walls), the sum running over the interior unknowns
// listed in cq (their coarse-level offsets in cx); ghosts are written with
// the stream BCs.
__global__ void k_coarse_apply(Lay L, const double* __restrict__ Ainv, const double* __restrict__ rowb,
                               const double* rhs, int n, const int* __restrict__ cq, const int* __restrict__ cx,
                               int m, double* err, int Vbc) {
    pdl_entry();
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= m) return;
    const int pw = __ldg(cq + w), N = L.b + 1;
    const double* row = Ainv + (size_t)pw * n;
    double acc = 0.0;
    for (int e = lane; e < m; e += 32) {
        const int q = __ldg(cq + e);
        acc = fma(__ldg(row + q), ld_state(rhs + __ldg(cx + e)) * __ldg(rowb + q), acc);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if (lane == 0) store_stream(L, err, pw / N, pw % N, acc, Vbc);
    pdl_done();
}
void launch_coarse_apply(cudaStream_t s, const Level& lv, const double* Ainv, const double* rowb, int n,
                         const int* cq, const int* cx, int m, double* err, int Vbc) {
    const int threads = 256;
    const unsigned nb = (unsigned)((m * 32 + threads - 1) / threads);
    launch_pdl(k_coarse_apply, nb, threads, 0, s, lv.L, Ainv, rowb, lv.rhs, n, cq, cx, m, err, Vbc); tc_note_launch();
}

// Coarsest-level solve for coarse grids too large for an explicit inverse:
// B = RowB .* RHS (Compute_coarse_vector), DGBTRS('N') with the band's LU
// (row interchanges + unit-lower solve, then dtbsv), x to the interior
// (Stream_grid_coarse with the stream BCs).  One cluster, the vector in the shared
// memory of its first CTA; every element sees DGBTRS's operations in its order.
//  - Forward, the first CTA: a row in reach per thread, re-based every 16 steps, the
//    band's columns loaded four steps ahead, one barrier a step.
//  - Backward, 32 rows at a time: a warp solves the block, one row per lane, and a second
//    follows it with the next block's rows, so that it can go on from there (they take
//    turns); meanwhile warps of the other CTAs apply the last block to the rows above.
// What bounds it is the chain of FP64 operations: a warp's takes 64 cycles, whether it
// depends on the one before or not, so the chain's warps share no scheduler with other
// FP64 work.  Forward 620 cycles a step (two operations of two warps, exchange, barrier),
// backward 720 (six operations, two of them the product with the pivot's reciprocal that
// replaces most of a division).  Against one warp doing every step on the vector in shared
// memory, at n = 10201, kl = 202: 27 -> 7.3 ms.
#define CS_THREADS 256
#define CS_CL 8
#define CS_MAXKL 496
#define CS_WAIT (1 << 20)  // polls of a wait for four solved rows
#define CS_TEST_WAIT (1 << 14)  // polls of the timeout-path test's word
template <typename TR, int RR>
__global__ void __launch_bounds__(CS_THREADS) k_coarse_solve(Lay L, const double* __restrict__ ABg,
                                                             const int* __restrict__ ipiv,
                                                             const double* __restrict__ rowb, const TR* rhs, int n,
                                                             int kl, int ku, TR* err, int Vbc, int* timeout_flag,
                                                             const int* test_flag) {
    constexpr int NP = 16, D = 4;  // steps between re-basings, steps loaded ahead
    extern __shared__ double Bv[];
    __shared__ double s_d[32], s_y[32], s_y2[32];  // pivots of a block and their reciprocals
    __shared__ __align__(8) unsigned long long bar[8];
    pdl_entry();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nzc = L.b, nxc = L.a, N = nzc + 1;
    const int ldab = 2 * kl + ku + 1, KD = ku + kl + 1, K = kl + ku;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    if (tid < 8) mbar_init(smem_addr(&bar[tid]), 32);
    for (int q = tid; rank == 0 && q < n; q += CS_THREADS) {
        const int kq = q % N, iq = q / N;
        Bv[q] = (iq >= 1 && iq <= nxc - 1 && kq >= 1 && kq <= nzc - 1)
                    ? (double)ld_state(rhs + IX(L, iq, kq)) * __ldg(rowb + q)
                    : 0.0;
    }
    __syncthreads();
    auto nonzero = [](double x) { return (unsigned long long)(__double_as_longlong(x) << 1) != 0ull; };
#define A_(rw, cl) ABg[(size_t)((rw) - 1) + (size_t)((cl) - 1) * ldab]
    if (rank == 0) {
        // rows b0 + o of the 16 steps from b0 on, o = tid + CS_THREADS u; column k's entry of row
        // b0 + o is in f, loaded D steps before
        double v[RR], f[D][RR];
        int piv[D];
        const double* from = &A_(KD + tid, 1);  // of the next fetch
        int kf = 1;
        auto fetch = [&](double(&g)[RR], int& p) {
            const int i = (kf - 1) & (NP - 1), KM = min(kl, n - kf);
            if (kf < n) p = __ldg(ipiv + kf - 1) - (kf - i);
#pragma unroll
            for (int u = 0; u < RR; u++) {
                const int t = tid + CS_THREADS * u - i;
                g[u] = (t >= 1 && t <= KM) ? __ldg(from + CS_THREADS * u) : 0.0;
            }
            from += i == NP - 1 ? ldab + NP - 1 : ldab - 1;
            kf++;
        };
#pragma unroll
        for (int q = 0; q < D; q++) {
            piv[q] = 0;
            fetch(f[q], piv[q]);
        }
        for (int b0 = 1; b0 < n; b0 += NP) {
#pragma unroll
            for (int u = 0; u < RR; u++) {
                const int r = b0 + tid + CS_THREADS * u;
                v[u] = r <= n ? Bv[r - 1] : 0.0;
            }
#pragma unroll 1
            for (int i0 = 0; i0 < NP && b0 + i0 < n; i0 += D) {
#pragma unroll
                for (int q = 0; q < D; q++) {
                    const int i = i0 + q, KM = min(kl, n - b0 - i), op = piv[q];
                    double* ex = s_d + 2 * (q & 1);
                    if (b0 + i < n) {
#pragma unroll
                        for (int u = 0; u < RR; u++)
                            if (tid + CS_THREADS * u == op) ex[0] = v[u];
                        if (tid == i) ex[1] = v[0];
                        __syncthreads();
                        const double top = ex[0], old = ex[1], temp = -top;
#pragma unroll
                        for (int u = 0; u < RR; u++) {
                            const int o = tid + CS_THREADS * u, t = o - i;
                            if (o == op) v[u] = old;
                            if (o == i) v[u] = top;
                            if (nonzero(temp) && t >= 1 && t <= KM) v[u] = v[u] + f[q][u] * temp;
                        }
                    }
                    fetch(f[q], piv[q]);
                }
            }
#pragma unroll
            for (int u = 0; u < RR; u++) {
                const int r = b0 + tid + CS_THREADS * u;
                if (r <= n) Bv[r - 1] = v[u];
            }
            __syncthreads();
        }
    }
    cl.sync();
    double* B0 = cl.map_shared_rank(Bv, 0);
    // the warp's rows: e - 32 - 32 g - lane, or e - lane where it solves.  Warps 0 and 1
    // of CTA 0 take turns at that; the other follows with the next block, g = 0
    const int g = rank + (CS_CL - 1) * warp;
    const bool far = rank > 0 && g <= (K - 1) / 32;
    // a block's columns at row e - 32 - 32 g - lane
    double f[32];
    auto fetch = [&](int e, int g) {
        const int i = e - 32 - 32 * g - lane;
        const double* from = &A_(K + 1 + i - e, e);
#pragma unroll
        for (int l = 0; l < 32; l++) {
            f[l] = (i >= 1 && e - l - i <= K) ? __ldg(from) : 0.0;
            from -= ldab - 1;
        }
    };
    double v = 0.0;  // of the chain: lane l has row e - l
    double pivot = 1.0;
    bool dead = false;
    if (test_flag != nullptr && rank == 0) {
        if (lane == 0)
            for (int it = 0; *(volatile const int*)test_flag == 0 && it < CS_TEST_WAIT; it++) {
            }
        dead = true;
    }
    if (rank == 0 && warp == 0) {
        if (n - lane >= 1) {
            v = Bv[n - lane - 1];
            pivot = __ldg(&A_(K + 1, n - lane));
        }
    }
    if (far) fetch(n, g);
    for (int e = n, it = 0; e >= 1; e -= 32, it++) {
        const int i = e - lane, i2 = i - 32;
        if (rank == 0 && warp == (it & 1)) {
            s_d[lane] = pivot;
            solve_recip(pivot, s_y[lane], s_y2[lane]);
            __syncwarp();
            // the block's columns, four steps ahead: column e - l at row i
            double a[4];
            const double* from = &A_(K + 1 - lane, e);
            auto near = [&](int l) {
                const double x = (lane > l && i >= 1 && lane - l <= K) ? __ldg(from) : 0.0;
                from -= ldab - 1;
                return x;
            };
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = near(q);
#pragma unroll 1
            for (int l0 = 0; l0 < 32; l0 += 4) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int l = l0 + q;
                    const double bj = __shfl_sync(0xffffffffu, v, l);
                    const double temp = solve_quot(bj, s_d[l], s_y[l], s_y2[l]);
                    const double w = v - temp * a[q];
                    v = nonzero(bj) && lane > l && lane - l <= K ? w : v;  // rows below the first are zero
                    if (nonzero(bj) && lane == l) v = temp;
                    a[q] = l + 4 < 32 ? near(l + 4) : 0.0;
                }
                if (lane >= l0 && lane < l0 + 4 && i >= 1) Bv[i - 1] = v;
                mbar_arrive(smem_addr(&bar[l0 / 4]));
            }
        }
        if (it > 0) cluster_wait();  // the block before is applied everywhere
        if (rank == 0 && warp == (~it & 1)) {
            v = i2 >= 1 ? Bv[i2 - 1] : 0.0;
            pivot = i2 >= 1 ? __ldg(&A_(K + 1, i2)) : 1.0;
            fetch(e, 0);
#pragma unroll
            for (int l0 = 0; l0 < 32; l0 += 4) {
                int spins = 0;
                while (!dead && !mbar_try_wait(smem_addr(&bar[l0 / 4]), it & 1)) dead = ++spins > CS_WAIT;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int l = l0 + q;
                    const double temp = e - l >= 1 ? Bv[e - l - 1] : 0.0;
                    const double w = v - temp * f[l];
                    v = (nonzero(temp) && i2 >= 1 && lane + 32 - l <= K) ? w : v;
                }
            }
        }
        cluster_arrive();
        cluster_wait();  // this block is solved
        const int r = i2 - 32 * g;
        if (far) {
            const double temps = i >= 1 ? B0[i - 1] : 0.0;
            double w = r >= 1 ? B0[r - 1] : 0.0;
#pragma unroll
            for (int l = 0; l < 32; l++) {
                const double temp = __shfl_sync(0xffffffffu, temps, l);
                const double x = w - temp * f[l];
                w = (nonzero(temp) && 32 + 32 * g + lane - l <= K) ? x : w;
            }
            if (r >= 1) B0[r - 1] = w;
            fetch(e - 32, g);
        }
        cluster_arrive();
    }
    cluster_wait();
    if (dead) atomicExch(timeout_flag, 1);
    if (rank != 0) return;
#undef A_
    for (int q = tid; q < n; q += CS_THREADS) {
        const int kq = q % N, iq = q / N;
        if (iq >= 1 && iq <= nxc - 1 && kq >= 1 && kq <= nzc - 1) store_stream<TR>(L, err, iq, kq, (TR)Bv[q], Vbc);
    }
    pdl_done();
}
// The same with one warp and no rows in registers: bands and vectors beyond the kernel
// above (kl > 496, or a vector that leaves no room for the pivots), and devices that do
// not take its cluster.
template <typename TR>
__global__ void __launch_bounds__(256) k_coarse_solve_wide(Lay L, const double* __restrict__ ABg,
                                                           const int* __restrict__ ipiv,
                                                           const double* __restrict__ rowb, const TR* rhs, int n,
                                                           int kl, int ku, TR* err, int Vbc) {
    extern __shared__ double Bv[];
    pdl_entry();
    const int tid = threadIdx.x, lane = tid & 31;
    const int nzc = L.b, nxc = L.a, N = nzc + 1;
    const int ldab = 2 * kl + ku + 1, KD = ku + kl + 1, K = kl + ku;
    for (int q = tid; q < n; q += blockDim.x) {
        const int kq = q % N, iq = q / N;
        Bv[q] = (iq >= 1 && iq <= nxc - 1 && kq >= 1 && kq <= nzc - 1)
                    ? (double)ld_state(rhs + IX(L, iq, kq)) * __ldg(rowb + q)
                    : 0.0;
    }
    __syncthreads();
#define A_(rw, cl) ABg[(size_t)((rw) - 1) + (size_t)((cl) - 1) * ldab]
    if (tid < 32) {
        for (int jj = 1; jj <= n - 1; jj++) {
            const int LM = min(kl, n - jj);
            const int Lr = __ldg(ipiv + jj - 1);
            if (Lr != jj) {
                if (lane == 0) { const double t0 = Bv[Lr - 1]; Bv[Lr - 1] = Bv[jj - 1]; Bv[jj - 1] = t0; }
                __syncwarp();
            }
            const double temp = -Bv[jj - 1];
            if (temp != 0.0)
                for (int t = 1 + lane; t <= LM; t += 32) Bv[jj + t - 1] = Bv[jj + t - 1] + __ldg(&A_(KD + t, jj)) * temp;
            __syncwarp();
        }
        for (int jj = n; jj >= 1; jj--) {
            const double bj = Bv[jj - 1];
            if (bj != 0.0) {
                const int Lc = K + 1 - jj;
                const double temp = bj / __ldg(&A_(K + 1, jj));
                __syncwarp();
                if (lane == 0) Bv[jj - 1] = temp;
                for (int i = jj - 1 - lane; i >= max(1, jj - K); i -= 32) Bv[i - 1] = Bv[i - 1] - temp * __ldg(&A_(Lc + i, jj));
            }
            __syncwarp();
        }
    }
#undef A_
    __syncthreads();
    for (int q = tid; q < n; q += blockDim.x) {
        const int kq = q % N, iq = q / N;
        if (iq >= 1 && iq <= nxc - 1 && kq >= 1 && kq <= nzc - 1) store_stream<TR>(L, err, iq, kq, (TR)Bv[q], Vbc);
    }
    pdl_done();
}
template <typename TR>
static void coarse_solve(cudaStream_t s, const Level& lv, const double* band, const int* ipiv, const double* rowb,
                         const TR* rhs, int n, int kl, int ku, TR* err, int Vbc, int* timeout_flag,
                         const int* test_flag) {
    const size_t sm = sizeof(double) * (size_t)n;
    auto go = [&](auto kernel, int ctas, auto... more) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas, 1, 1);
        cfg.blockDim = dim3(CS_THREADS, 1, 1);
        cfg.dynamicSmemBytes = sm;
        cfg.stream = s;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = ctas;
        at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = ctas > 1 ? 2 : 1;
        if ((ctas > 1 && lv.no_cluster) ||
            cudaLaunchKernelEx(&cfg, kernel, lv.L, band, ipiv, rowb, rhs, n, kl, ku, err, Vbc, more...) != cudaSuccess)
            return false;
        tc_note_launch();
        return true;
    };
    // two rows per thread above kl = 240: the 16 steps between re-basings reach kl + 16 rows
    if (kl <= CS_MAXKL && sm <= 226 * 1024) {
        if (kl <= 240 ? go(k_coarse_solve<TR, 1>, CS_CL, timeout_flag, test_flag)
                      : go(k_coarse_solve<TR, 2>, CS_CL, timeout_flag, test_flag)) return;
        cudaGetLastError();
    }
    go(k_coarse_solve_wide<TR>, 1);  // (an error here is left for the solve's next read)
}
void launch_coarse_solve(cudaStream_t s, const Level& lv, const double* band, const int* ipiv, const double* rowb,
                         int n, int kl, int ku, double* err, int Vbc, int* timeout_flag, const int* test_flag) {
    coarse_solve(s, lv, band, ipiv, rowb, (const double*)lv.rhs, n, kl, ku, err, Vbc, timeout_flag, test_flag);
}
void launch_coarse_solve32(cudaStream_t s, const Level& lv, const double* band, const int* ipiv, const double* rowb,
                           int n, int kl, int ku, float* err, int Vbc, int* timeout_flag, const int* test_flag) {
    coarse_solve(s, lv, band, ipiv, rowb, (const float*)lv.rhs32, n, kl, ku, err, Vbc, timeout_flag, test_flag);
}

__global__ void k_copy(double* dst, const double* src, size_t n) {
    pdl_entry();
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t st = (size_t)gridDim.x * blockDim.x;
    for (; t < n; t += st) dst[t] = ld_state(src + t);
    pdl_done();
}
void launch_copy_plane(cudaStream_t s, double* dst, const double* src, size_t n) {
    int nb = (int)((n + 255) / 256);
    if (nb > 1216) nb = 1216;
    launch_pdl(k_copy, nb, 256, 0, s, dst, src, n); tc_note_launch();
}

// compute_RHS(1) and compute_reference_residual(1)
__global__ void k_rhs1(Lay L, Phys P, Range2 r, const double* __restrict__ Tb, CPtrs Cb, double* __restrict__ rhs,
                       RedScratch rs, double* out, double div1, double div2) {
    RANGE_IK(r);
    double a = 0.0;
    if (inr) {
        size_t x = IX(L, i, k);
        double R = 0.0;
        // dx/dr at node i (1 on a uniform grid, where the division is skipped)
        const double x1 = P.M.on ? mt(P.M.xr, i) : 1.0;
        if (P.RaT != 0.0) {
            double Tr = first_diff(Tb[x - 1], Tb[x + 1], P.dr, P.rdr, P.dr_pow2);
            if (P.M.on) Tr = Tr / x1;
            R = P.RaT * Tr;
        }
        if (P.comp == 1)
            for (int j = 0; j < P.ntype; j++) {
                double Cr = first_diff(Cb.p[j][x - 1], Cb.p[j][x + 1], P.dr, P.rdr, P.dr_pow2);
                if (P.M.on) Cr = Cr / x1;
                R = R - P.RaC[j] * Cr;
            }
        rhs[x] = R;
        a = fabs(R);
    }
    reduce_to(RED_SUM, a, rs.part, rs.count, out, div1, div2);
}
void launch_rhs1(cudaStream_t s, const Lay& L, const Phys& P, const double* Tbuoy, const double* const* Cbuoy,
                 double* rhs, RedScratch rs, DevScalars* ds) {
    Range2 r{1, L.a - 1, 1, L.b - 1};
    CPtrs C{};
    for (int j = 0; j < P.ntype && j < TC_MAX_TYPES; j++) C.p[j] = Cbuoy[j];
    k_rhs1<<<grid_for(r), dim3(BX, BY), 0, s>>>(L, P, r, Tbuoy, C, rhs, rs, &ds->res_ref, (double)(L.a - 2),
                                                 (double)(L.b - 2)); tc_note_launch();
}
