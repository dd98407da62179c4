// The single-component boundary cells' kernel.
#pragma once
#include "sc_kernels.cuh"

namespace lbm {

// ----------------------------------------------------------------------------------
// The special cells: streaming (reference LBM::Streaming, src/lbm-streaming.cpp:3-119: bounce-back
// off solid (f only) and adiabatic (f and g) cells, specular reflection off free-slip cells
// (dirSlip, src/lbm-bc.cpp:1352-1399), populations kept along inflow/outflow directions and g along
// solid ones, periodic wrap otherwise), the Tamm-Mott-Smith boundary treatment (LBM::TMS_BC, single
// component: outflow src/lbm-bc.cpp:341-460, inflow :809-938, solid :1111-1229, in that order) and
// the moments.
//
// A block of two warps per 32 listed cells: lane = cell, warp = set (f, g).  A thread holds its set's
// 27 populations and one set of per-axis factors in registers; the sums of one set that the other
// needs go through shared memory.  The target and local sets are not stored: each sweep over the
// directions forms them from the factors.  What bounds it is the chain of one cell's operations (one
// thread per cell held 27 x 6 values, spilled, and looked up 27 neighbour types for every sweep).
// Measured with the 97 x 41 x 30 channel's 8,160 special cells: 50 us after the interior's kernel, now
// 30 us beside it (the step 98 -> 61 us); what is left is mostly instruction fetch, so both warps
// run one copy of the equilibrium's code and the passes and sweeps are rolled loops (40 us with
// a copy per set).
// ----------------------------------------------------------------------------------
constexpr int kScSpCells = 32;
struct ScSpSmem {
    double x[2][5][kScSpCells];  // exchanged sums, two generations: rho, j (3), rhoE
    unsigned up[7][kScSpCells];  // directions with an upstream cell of each kind
    uint8_t dir[27];             // dir_code, for a direction known at run time only
};
enum : int { SU_OUT = 0, SU_IN = 1, SU_KEEP = 2, SU_SOLID = 3, SU_ADI = 4, SU_SLIP = 5, SU_FLUID = 6 };

__global__ void __launch_bounds__(2 * kScSpCells)
    k_sc_special(ScGeom g, ScPhys P, const int8_t *__restrict__ type, const long *__restrict__ blist,
                 const double *__restrict__ pop, const double *__restrict__ mom, double *__restrict__ mom_nxt,
                 const double *__restrict__ bst_cur, double *__restrict__ bst_nxt, long nb, unsigned *status) {
    __shared__ ScSpSmem sm;
    const int lane = threadIdx.x & 31, set = threadIdx.x >> 5;
    const long b0 = (long)blockIdx.x * kScSpCells + lane, nc = g.ncell;
    const bool valid = b0 < nb;  // a lane past the list's end takes the last cell and stores nothing
    const long b = valid ? b0 : nb - 1, n = blist[b];
    int i, j, k;
    cell_ijk(n, g.si, g.sj, i, j, k);
    for (int q = set; q < 7; q += 2) sm.up[q][lane] = 0u;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int l = 0; l < 27; ++l) sm.dir[l] = dir_code(l);
    }
    __syncthreads();
    auto offset = [&](int l) {
        const unsigned c = sm.dir[l];
        return (long)dec2(c & 3) * g.si + (long)dec2((c >> 2) & 3) * g.sj + dec2((c >> 4) & 3);
    };
    int ty[14];  // the warp's directions 2 q + set, all loads before the first use
#pragma unroll
    for (int q = 0; q < 14; ++q) {
        const unsigned c = set && q < 13 ? dir_code(q < 13 ? 2 * q + 1 : 26) : dir_code(2 * q);
        ty[q] = type[n - ((long)dec2(c & 3) * g.si + (long)dec2((c >> 2) & 3) * g.sj + dec2((c >> 4) & 3))];
    }
#pragma unroll
    for (int q = 0; q < 14; ++q) {
        const int l = 2 * q + set, t = ty[q];
        if (l > 26) continue;
        const unsigned m = 1u << l;
        if (t == T_O) atomicOr(&sm.up[SU_OUT][lane], m);
        if (t == T_I) atomicOr(&sm.up[SU_IN][lane], m);
        if (t == T_O || t == T_O_C || t == T_I || t == T_I_C) atomicOr(&sm.up[SU_KEEP][lane], m);
        if (t == T_S) atomicOr(&sm.up[SU_SOLID][lane], m);
        if (t == T_A) atomicOr(&sm.up[SU_ADI][lane], m);
        if (t == T_FS) atomicOr(&sm.up[SU_SLIP][lane], m);
        if (t == T_F) atomicOr(&sm.up[SU_FLUID][lane], m);
    }
    __syncthreads();
    const unsigned out_m = sm.up[SU_OUT][lane], in_m = sm.up[SU_IN][lane], sol_m = sm.up[SU_SOLID][lane],
                   slip_m = sm.up[SU_SLIP][lane], fluid_up = sm.up[SU_FLUID][lane];
    // fluid downstream along l: fluid upstream along opp(l) (opposite directions are neighbours)
    const unsigned fluid_dn = (fluid_up & 1u) | ((fluid_up & 0x2aaaaaau) << 1) | ((fluid_up & 0x5555554u) >> 1);

    double f[27];
    {
        const unsigned kept_m = sm.up[SU_KEEP][lane] | (set ? sol_m : 0u),
                       back_m = (sol_m | sm.up[SU_ADI][lane]) & ~kept_m;
        PullSrc ps;
        pull_src(g, i, j, k, ps);
#pragma unroll
        for (int l = 0; l < 27; ++l) {
            const bool kept = (kept_m >> l) & 1, back = (back_m >> l) & 1;
            const long at = back || ((slip_m >> l) & 1) ? n : (long)pull_at(ps, l);
            f[l] = kept ? bst_cur[(long)(27 * set + l) * nb + b] : pop[(long)(27 * set + (back ? opp(l) : l)) * nc + at];
        }
        if (slip_m) {
#pragma unroll
            for (int l = 1; l < 27; ++l) {
                if (!((slip_m >> l) & 1)) continue;
                int in = i - cx(l), jn = j - cy(l), kn = k - cz(l), lp = l;
                if (cx(l) && ((slip_m >> dir3(cidx(cx(l)), 0, 0)) & 1)) {
                    lp = dir3(cidx(-cx(l)), cidx(cy(l)), cidx(cz(l)));
                    in = i;
                } else if (cy(l) && ((slip_m >> dir3(0, cidx(cy(l)), 0)) & 1)) {
                    lp = dir3(cidx(cx(l)), cidx(-cy(l)), cidx(cz(l)));
                    jn = j;
                } else if (cz(l) && ((slip_m >> dir3(0, 0, cidx(cz(l)))) & 1)) {
                    lp = dir3(cidx(cx(l)), cidx(cy(l)), cidx(-cz(l)));
                    kn = k;
                }
                in = ((in - 1 + (g.Nx - 2)) % (g.Nx - 2)) + 1;
                jn = ((jn - 1 + (g.Ny - 2)) % (g.Ny - 2)) + 1;
                kn = ((kn - 1 + (g.Nz - 2)) % (g.Nz - 2)) + 1;
                f[l] = pop[(long)(27 * set + lp) * nc + (long)in * g.si + (long)jn * g.sj + kn];
            }
        }
    }
    int gen = 0;
    auto flip = [&] {
        __syncthreads();
        gen ^= 1;
    };
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
        const unsigned bm = pass == 0 ? out_m : (pass == 1 ? in_m : sol_m), fm = bm & fluid_dn;
        const bool on = fm != 0;
        if (!__syncthreads_or(on)) continue;
        // the target's density, velocity and temperature
        double rho_t, vel_t[3], T_t;
        if (pass < 2) {  // the first direction with the type upstream and fluid downstream
            const long o = on ? offset(__ffs((int)fm) - 1) : 0, ni = n + o, ng = n - o;
            const long nv = pass == 0 ? ni : ng, np = pass == 0 ? ng : ni;
#pragma unroll
            for (int d = 0; d < 3; ++d) vel_t[d] = mom[(M_U + d) * nc + nv];
            T_t = mom[M_T * nc + nv];
            rho_t = mom[M_P * nc + np] / (P.R * T_t);
        } else {  // half-way interpolated target, q = 0.5
            const double q = 0.5;
            vel_t[0] = vel_t[1] = vel_t[2] = T_t = 0.0;
            for (unsigned mm = fm; mm; mm &= mm - 1) {
                const long o = offset(__ffs((int)mm) - 1);
#pragma unroll
                for (int d = 0; d < 3; ++d) vel_t[d] += q * mom[(M_U + d) * nc + n + o] + mom[(M_U + d) * nc + n - o];
                T_t += q * mom[M_T * nc + n + o] + mom[M_T * nc + n - o];
            }
            const double inv = 1.0 / ((1.0 + q) * (on ? __popc(fm) : 1));
#pragma unroll
            for (int d = 0; d < 3; ++d) vel_t[d] = inv * vel_t[d];
            T_t = inv * T_t;
            double r = 0.0;
#pragma unroll
            for (int l = 0; l < 27; ++l) r += f[l];
            if (set == 0) sm.x[gen][0][lane] = r;
            flip();
            rho_t = sm.x[gen ^ 1][0][lane];
        }
        // outflow, solid: f = (2 f_t | f + f_t) - f_loc; inflow: f = (f_t | f) + f_new - f_loc with f_new
        // the target at the local density
        double rho_x = rho_t, vel_x[3] = {vel_t[0], vel_t[1], vel_t[2]}, T_x = T_t, rho_l = 0.0, vel_l[3], T_l = 0.0;
#pragma unroll 1
        for (int stage = 0; stage < 3; ++stage) {
            if (stage == 1 && pass != 1) continue;
            // the energy set's equilibrium as B p_z + C A_z per pair (c_x, c_y); with E = 1 and A = 0 it is the
            // product form of f, so both warps run the same code
            AxisG<double> G;
            axis_geq(G, P.cv * T_x, P.R * T_x, vel_x);
            if (set == 0) {
                G.E = 1.0;
#pragma unroll
                for (int a = 0; a < 3; ++a) G.A[a][0] = G.A[a][1] = G.A[a][2] = 0.0;
            }
            double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int ix = 0; ix < 3; ++ix) {
                const double px = rho_x * G.P[0][ix], tx = rho_x * (G.E * G.P[0][ix] + G.A[0][ix]);
#pragma unroll
                for (int iy = 0; iy < 3; ++iy) {
                    const double B = tx * G.P[1][iy] + px * G.A[1][iy], C = px * G.P[1][iy];
#pragma unroll
                    for (int iz = 0; iz < 3; ++iz) {
                        const int l = dir3(ix, iy, iz);
                        const double e = B * G.P[2][iz] + C * G.A[2][iz];
                        const bool bd = (bm >> l) & 1;
                        if (stage == 0) {
                            const double fv = bd ? e : f[l];
                            s[0] += fv;
                            if (cx(l)) s[1] += cx(l) * fv;
                            if (cy(l)) s[2] += cy(l) * fv;
                            if (cz(l)) s[3] += cz(l) * fv;
                            if (on) f[l] = pass == 1 ? fv : (bd ? 2 * e : e + f[l]);
                        } else if (on) {
                            f[l] = stage == 1 ? e + f[l] : f[l] - e;
                        }
                    }
                }
            }
            if (stage == 0) {  // the local state and its temperature
                if (set == 0) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) sm.x[gen][q][lane] = s[q];
                } else {
                    sm.x[gen][4][lane] = s[0];
                }
                flip();
                const double(*x)[kScSpCells] = sm.x[gen ^ 1];
                rho_l = x[0][lane];
#pragma unroll
                for (int d = 0; d < 3; ++d) vel_l[d] = x[1 + d][lane] / rho_l;
                T_l = (x[4][lane] / rho_l - 0.5 * (vel_l[0] * vel_l[0] + vel_l[1] * vel_l[1] + vel_l[2] * vel_l[2])) / P.cv;
            }
            const bool fresh = stage == 0 && pass == 1;
            rho_x = rho_l;
            T_x = fresh ? T_t : T_l;
#pragma unroll
            for (int d = 0; d < 3; ++d) vel_x[d] = fresh ? vel_t[d] : vel_l[d];
        }
    }
    if (valid) {
#pragma unroll
        for (int l = 0; l < 27; ++l) bst_nxt[(long)(27 * set + l) * nb + b] = f[l];
    }
    if (set == 1) {
        double e = 0.0;
#pragma unroll
        for (int l = 0; l < 27; ++l) e += f[l];
        sm.x[gen][4][lane] = e;
    }
    __syncthreads();
    if (set == 1 || !valid) return;
    ScSums s;
    sums_init(s);
#pragma unroll
    for (int l = 0; l < 27; ++l) sums_add(s, l, f[l], 0.0);
    s.re = sm.x[gen][4][lane];
    store_record_sc(g, P, n, s, mom_nxt, status);
}

}  // namespace lbm
