// The single-component boundary cells' kernel.
#pragma once
#include "sc_kernels.cuh"

namespace lbm {

// Specular partner of direction l off a free-slip neighbour (reference LBM::dirSlip,
// src/lbm-bc.cpp:1352-1399).
__device__ __forceinline__ void dir_slip(const ScGeom &g, const int8_t *__restrict__ type, int l, int i, int j,
                                         int k, int &lp, long &src) {
    const int inb = i - cx(l), jnb = j - cy(l), knb = k - cz(l);
    int cxp = cx(l), cyp = cy(l), czp = cz(l);
    int ip = inb, jp = jnb, kp = knb;
    if (type_at(g, type, inb, j, k) == T_FS) {
        cxp = -cxp;
        ip = i;
    } else if (type_at(g, type, i, jnb, k) == T_FS) {
        cyp = -cyp;
        jp = j;
    } else if (type_at(g, type, i, j, knb) == T_FS) {
        czp = -czp;
        kp = k;
    }
    ip = ((ip - 1 + (g.Nx - 2)) % (g.Nx - 2)) + 1;
    jp = ((jp - 1 + (g.Ny - 2)) % (g.Ny - 2)) + 1;
    kp = ((kp - 1 + (g.Nz - 2)) % (g.Nz - 2)) + 1;
    lp = l;
#pragma unroll
    for (int a = 0; a < 27; ++a)
        if (cx(a) == cxp && cy(a) == cyp && cz(a) == czp) lp = a;
    src = (long)ip * g.si + (long)jp * g.sj + kp;
}

// Streaming of a special cell (reference LBM::Streaming, src/lbm-streaming.cpp:3-119):
// bounce-back off solid (f only) and adiabatic (f and g) cells, specular reflection off
// free-slip cells, populations kept (`stale`) along inflow/outflow directions, periodic
// wrap otherwise.
__device__ __forceinline__ void pull_special(const ScGeom &g, const int8_t *__restrict__ type, long n,
                                             const double *__restrict__ pop, const double *__restrict__ stale,
                                             long nb_stride, double f[27], double ge[27]) {
    const long nc = g.ncell;
    int i, j, k;
    cell_ijk(n, g.si, g.sj, i, j, k);
#pragma unroll
    for (int l = 0; l < 27; ++l) {
        int in = i - cx(l), jn = j - cy(l), kn = k - cz(l);
        const int tn = type_at(g, type, in, jn, kn);
        if (tn == T_S) {
            f[l] = pop[(long)opp(l) * nc + n];
            ge[l] = stale[(long)(27 + l) * nb_stride];
        } else if (tn == T_FS) {
            int lp;
            long src;
            dir_slip(g, type, l, i, j, k, lp, src);
            f[l] = pop[(long)lp * nc + src];
            ge[l] = pop[(long)(27 + lp) * nc + src];
        } else if (tn == T_A) {
            f[l] = pop[(long)opp(l) * nc + n];
            ge[l] = pop[(long)(27 + opp(l)) * nc + n];
        } else if (tn == T_O || tn == T_O_C || tn == T_I || tn == T_I_C) {
            f[l] = stale[(long)l * nb_stride];
            ge[l] = stale[(long)(27 + l) * nb_stride];
        } else {
            if (in == 0) in = g.Nx - 2; else if (in == g.Nx - 1) in = 1;
            if (jn == 0) jn = g.Ny - 2; else if (jn == g.Ny - 1) jn = 1;
            if (kn == 0) kn = g.Nz - 2; else if (kn == g.Nz - 1) kn = 1;
            const long s = (long)in * g.si + (long)jn * g.sj + kn;
            f[l] = pop[(long)l * nc + s];
            ge[l] = pop[(long)(27 + l) * nc + s];
        }
    }
}

// Target populations of a prescribed (rho, u, T) (reference calculate_feq_geq,
// src/lbm-edf.cpp:153-164).
__device__ __forceinline__ void target_sc(const ScPhys &P, double rho, const double vel[3], double T, double ft[27],
                                          double gt[27]) {
    const double theta = P.R * T;
    const double zero[3] = {0.0, 0.0, 0.0};
    AxisF<double> F;
    axis_feq(F, vel, theta, zero);
    AxisG<double> G;
    axis_geq(G, P.cv * T, theta, vel);
#pragma unroll
    for (int l = 0; l < 27; ++l) {
        ft[l] = feq_l(l, rho, F);
        gt[l] = geq_l(l, rho, G);
    }
}

// Local state of the cell with boundary directions (upstream type `bt`) replaced by the
// target set, and its temperature (src/lbm-bc.cpp:381-410, 874-903, 1167-1196).
__device__ __forceinline__ void local_state_sc(const ScGeom &g, const ScPhys &P, const int8_t *__restrict__ type, int i,
                                               int j, int k, int bt, const double f[27], const double ge[27],
                                               const double ft[27], const double gt[27], double &rho_o, double vel[3],
                                               double &T_o) {
    double rho = 0, ru = 0, rv = 0, rw = 0, re = 0;
#pragma unroll
    for (int l = 0; l < 27; ++l) {
        const bool b = type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == bt;
        const double fv = b ? ft[l] : f[l];
        const double gv = b ? gt[l] : ge[l];
        rho += fv;
        ru += fv * cx(l);
        rv += fv * cy(l);
        rw += fv * cz(l);
        re += gv;
    }
    vel[0] = ru / rho;
    vel[1] = rv / rho;
    vel[2] = rw / rho;
    const double Uint = re / rho - 0.5 * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
    T_o = Uint / P.cv;
    rho_o = rho;
}

// Tamm-Mott-Smith boundary treatment of one fluid cell (reference LBM::TMS_BC, single
// component: outflow src/lbm-bc.cpp:341-460, inflow :809-938, solid :1111-1229), applied
// in the reference's pass order.  `mom` holds the previous step's record.
static __device__ void tms_cell_sc(const ScGeom &g, const ScPhys &P, const int8_t *__restrict__ type,
                            const double *__restrict__ mom, long n, double f[27], double ge[27]) {
    const long nc = g.ncell;
    int i, j, k;
    cell_ijk(n, g.si, g.sj, i, j, k);
    double ft[27], gt[27], fl[27], gl[27];
    // ---- outflow: first direction with an outflow cell upstream and fluid downstream
    {
        int li = -1;
        long ni = n, ng = n;
#pragma unroll
        for (int l = 26; l >= 0; --l)
            if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_O &&
                type_at(g, type, i + cx(l), j + cy(l), k + cz(l)) == T_F) {
                li = l;
                ni = nb_index(g, n, cx(l), cy(l), cz(l));
                ng = nb_index(g, n, -cx(l), -cy(l), -cz(l));
            }
        if (li >= 0) {
            const double vel[3] = {mom[M_U * nc + ni], mom[M_V * nc + ni], mom[M_W * nc + ni]};
            const double T_out = mom[M_T * nc + ni];
            const double rho_out = mom[M_P * nc + ng] / (P.R * T_out);
            target_sc(P, rho_out, vel, T_out, ft, gt);
            double rl, vl[3], Tl;
            local_state_sc(g, P, type, i, j, k, T_O, f, ge, ft, gt, rl, vl, Tl);
            target_sc(P, rl, vl, Tl, fl, gl);
#pragma unroll
            for (int l = 0; l < 27; ++l) {
                if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_O) {
                    f[l] = 2 * ft[l] - fl[l];
                    ge[l] = 2 * gt[l] - gl[l];
                } else {
                    f[l] = ft[l] + f[l] - fl[l];
                    ge[l] = gt[l] + ge[l] - gl[l];
                }
            }
        }
    }
    // ---- inflow
    {
        int li = -1;
        long ni = n, ng = n;
#pragma unroll
        for (int l = 26; l >= 0; --l)
            if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_I &&
                type_at(g, type, i + cx(l), j + cy(l), k + cz(l)) == T_F) {
                li = l;
                ni = nb_index(g, n, cx(l), cy(l), cz(l));
                ng = nb_index(g, n, -cx(l), -cy(l), -cz(l));
            }
        if (li >= 0) {
            const double vin[3] = {mom[M_U * nc + ng], mom[M_V * nc + ng], mom[M_W * nc + ng]};
            const double T_in = mom[M_T * nc + ng];
            const double rho_in = mom[M_P * nc + ni] / (P.R * T_in);
            double fi[27], gi[27];
            target_sc(P, rho_in, vin, T_in, fi, gi);
            double rl, vl[3], Tl;
            local_state_sc(g, P, type, i, j, k, T_I, f, ge, fi, gi, rl, vl, Tl);
            target_sc(P, rl, vl, Tl, fl, gl);
            target_sc(P, rl, vin, T_in, ft, gt);
#pragma unroll
            for (int l = 0; l < 27; ++l) {
                if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_I) {
                    f[l] = ft[l] + fi[l] - fl[l];
                    ge[l] = gt[l] + gi[l] - gl[l];
                } else {
                    f[l] = ft[l] + f[l] - fl[l];
                    ge[l] = gt[l] + ge[l] - gl[l];
                }
            }
        }
    }
    // ---- solid walls, half-way interpolated target (q = 0.5)
    {
        int nd = 0;
        double vt[3] = {0, 0, 0}, Tt = 0;
        const double q = 0.5;
#pragma unroll
        for (int l = 0; l < 27; ++l) {
            if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_S &&
                type_at(g, type, i + cx(l), j + cy(l), k + cz(l)) == T_F) {
                const long hi = nb_index(g, n, cx(l), cy(l), cz(l));
                const long lo = nb_index(g, n, -cx(l), -cy(l), -cz(l));
                ++nd;
                vt[0] += (q * mom[M_U * nc + hi] + mom[M_U * nc + lo]) / (1.0 + q);
                vt[1] += (q * mom[M_V * nc + hi] + mom[M_V * nc + lo]) / (1.0 + q);
                vt[2] += (q * mom[M_W * nc + hi] + mom[M_W * nc + lo]) / (1.0 + q);
                Tt += (q * mom[M_T * nc + hi] + mom[M_T * nc + lo]) / (1.0 + q);
            }
        }
        if (nd > 0) {
            double rho_bb = 0;
#pragma unroll
            for (int l = 0; l < 27; ++l) rho_bb += f[l];
            const double inv = 1.0 / nd;
            vt[0] = inv * vt[0];
            vt[1] = inv * vt[1];
            vt[2] = inv * vt[2];
            Tt = inv * Tt;
            target_sc(P, rho_bb, vt, Tt, ft, gt);
            double rl, vl[3], Tl;
            local_state_sc(g, P, type, i, j, k, T_S, f, ge, ft, gt, rl, vl, Tl);
            target_sc(P, rl, vl, Tl, fl, gl);
#pragma unroll
            for (int l = 0; l < 27; ++l) {
                if (type_at(g, type, i - cx(l), j - cy(l), k - cz(l)) == T_S) {
                    f[l] = 2 * ft[l] - fl[l];
                    ge[l] = 2 * gt[l] - gl[l];
                } else {
                    f[l] = ft[l] + f[l] - fl[l];
                    ge[l] = gt[l] + ge[l] - gl[l];
                }
            }
        }
    }
}

__device__ __forceinline__ void sums_sc(const double f[27], const double ge[27], ScSums &s) {
    sums_init(s);
#pragma unroll
    for (int l = 0; l < 27; ++l) sums_add(s, l, f[l], ge[l]);
}

constexpr int kScSpBlock = 32;
// The special cells (compact list): streaming with bounce-back, free-slip and persisting populations, the
// TMS boundary treatment (reference LBM::TMS_BC), moments.  One thread per cell, bound by the chain of
// one cell's operations, so it runs beside the interior's kernel on the side stream, in blocks of 32
// threads that spread the list over the SMs.  The 97 x 41 x 30 channel's 8,160 cells: 53 us, now behind
// the interior's 17 us instead of after it (the step 100 -> 87 us).  A block of two warps per 32 cells
// (one per set, sums exchanged in shared memory) took 30 us, but rounded otherwise: the spanwise velocity,
// 1e-7 there, came out 1e-9 of itself away.
__global__ void __launch_bounds__(kScSpBlock)
    k_sc_special(ScGeom g, ScPhys P, const int8_t *__restrict__ type, const long *__restrict__ blist,
                               const double *__restrict__ src, const double *__restrict__ mom_cur,
                               double *__restrict__ mom_nxt, const double *__restrict__ bst_cur,
                               double *__restrict__ bst_nxt, long nb, unsigned *status) {
    const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const long n = blist[b];
    double f[27], ge[27];
    pull_special(g, type, n, src, bst_cur + b, nb, f, ge);
    tms_cell_sc(g, P, type, mom_cur, n, f, ge);
#pragma unroll
    for (int l = 0; l < 27; ++l) {
        bst_nxt[(long)l * nb + b] = f[l];
        bst_nxt[(long)(27 + l) * nb + b] = ge[l];
    }
    ScSums s;
    sums_sc(f, ge, s);
    store_record_sc(g, P, n, s, mom_nxt, status);
}

}  // namespace lbm
