// The boundary cells' kernel: streaming with the reference's per-type rules, the
// Tamm-Mott-Smith passes (characteristic outflow with NSCBC, inline LODI inflow, solid wall)
// and the moments of every cell with a boundary upstream -- mc_special_cell (mc_bc.cuh: the
// per-cell function, with the reference's file:line references, which the host build runs),
// the same operations in the same order, by a block of NS + 1 warps per 32 listed cells:
// lane = cell, warp = population set (species 0..NS-1, then the energy set).
//
// What bounds it: the chain of one cell's dependent FP64 operations, not bytes (a boundary
// layer holds a few thousand cells).  One thread per cell walked the 270 populations, the nine
// species' thermodynamics and the 9 x 9 Stefan-Maxwell system one after the other out of 5.7 kB
// of local memory.  Here a thread holds its own set's 27 populations in registers and its own
// species' part of every formula; the sums over the species are formed by every thread from
// the block's shared memory, in species order, so all warps hold the same bits and no
// result has to be sent back.  A cell that a pass does not concern, and a cell whose Newton
// iteration has ended, keeps its values while the block finishes the pass.
//
// Measured (B200, time of the kernel beside the interior's gather and solve): 8,256 cells of the
// 512 x 8 x 8 flame channel, FP32 storage, 436 -> 149 us (the step 785 -> 491 us); 3,840 cells of a
// 64 x 48 x 40 inflow layer, FP64, 494 -> 132 us (1041 -> 823 us); alone 110 and 62 us.  What is left is
// instruction fetch and the fixed latencies of one pass through the code by ten warps per SM; one copy of each
// part of the passes (the loops over pass and stage below) took 231 to 180 us.  The populations in
// shared memory with two blocks per SM (96 registers) was no faster (182 us there, 160 us for the
// inflow layer).
//
// This unit is compiled without fused multiply-adds (the Makefile): the boundary formulas lean on
// quantities that cancel exactly where the flow is uniform (target against local populations,
// one-sided differences), and an upwind switch downstream reads the sign of what is left.  With
// contraction the flame channel drifted 4e-9 from the reference in 20 steps, without it 3e-12.
#pragma once
#include "mc_bc.cuh"
#include "mc_cell.cuh"
#include "mc_moments.cuh"
#include "mc_ops.cuh"

namespace lbm {

constexpr int kSpCells = 32;  // cells of a block, one per lane
// kinds of upstream cells, each a mask over the 27 directions
enum : int { SP_OUT = 0, SP_IN = 1, SP_SOLID = 2, SP_ADI = 3, SP_SLIP = 4, SP_FLUID = 5, SP_MASKS = 6 };

template <int NS>
struct SpSmem {
    double x[2][4][NS + 1][kSpCells];  // exchanged values, two generations (see SpBlock::flip)
    double big[6 * NS][kSpCells];      // the species' P-tensor shares, then the Stefan-Maxwell factor
    double us[3][NS][kSpCells];        // species velocities
    unsigned up[SP_MASKS][kSpCells];   // directions with an upstream cell of each kind
    uint8_t dir[27];                   // dir_code, for a direction known at run time only
};

// A block's exchange of per-set values.  put() into the current generation, flip() (the block's
// barrier), then get(): the next put() goes to the other generation, so a slow reader of this one
// is never overtaken (a generation is rewritten only after another barrier).
template <int NS>
struct SpBlock {
    SpSmem<NS> &s;
    const int lane, set;
    int g;
    __device__ __forceinline__ void put(int q, double v) { s.x[g][q][set][lane] = v; }
    __device__ __forceinline__ void flip() {
        __syncthreads();
        g ^= 1;
    }
    __device__ __forceinline__ bool flip_any(bool v) {
        const bool any = __syncthreads_or(v);
        g ^= 1;
        return any;
    }
    __device__ __forceinline__ double get(int q, int a) const { return s.x[g ^ 1][q][a][lane]; }
    __device__ __forceinline__ double sum(int q) const {  // over the species, in their order
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < NS; ++a) v += get(q, a);
        return v;
    }
    __device__ __forceinline__ double sum_w(int q, const gas::Tables &t) const {  // with 1 / W_a
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < NS; ++a) v += get(q, a) * t.invW[a];
        return v;
    }
};

// set_mass_fractions with species a's share per thread: Y of the thread's species from its
// ratio y, returns the mean molar mass.
template <int NS>
__device__ __forceinline__ double sp_mass_fractions(SpBlock<NS> &B, const gas::Tables &t, double y, double &Y) {
    const double yc = y > 0.0 ? y : 0.0;
    B.put(0, yc);
    B.flip();
    Y = yc / B.sum(0);
    B.put(0, B.set < NS ? Y / t.m.W[B.set] : 0.0);
    B.flip();
    return 1.0 / B.sum(0);
}

// T_from_u / T_from_u_fast of the cells that are `on`, with the thread's species' share per
// iteration; the block iterates until its last cell has converged: by the moments' rule
// (MOMENTS, gas::newton_done), or to the local state's 1e-9.
template <int NS, bool FAST, bool MOMENTS>
__device__ __forceinline__ int sp_T_from_u(SpBlock<NS> &B, const gas::Tables &t, double Y, double u, double T0,
                                           bool on, double &T) {
    T = T0 > 0 ? T0 : 300.0;
    constexpr int maxit = 100;
    int it_used = on ? -1 : 0;
    const int a = B.set < NS ? B.set : NS - 1;
    for (int it = 0; it <= maxit; ++it) {
        if (FAST) {
            const double invT = 1.0 / T;
            B.put(0, Y * (gas::h_RT_fast(t, a, T, invT) - 1.0));
        } else {
            B.put(0, Y * (gas::h_RT_q(t, a, T) - 1.0));
        }
        B.put(1, Y * (gas::cp_R(t, a, T) - 1.0));
        // the last round only learns that no cell is left (or that the cap is reached)
        if (!B.flip_any(it_used < 0 && it < maxit)) break;
        if (it_used >= 0) continue;
        const double e = B.sum_w(0, t), c = B.sum_w(1, t);
        double dT;
        if (FAST) {
            dT = -(e * gas::kR * T - u) / (c * gas::kR);
        } else {
            const double f = e * gas::kR * T - u;
            const double cv = c * gas::kR;
            dT = -f / cv;
        }
        if (dT > 500.0) dT = 500.0;
        if (dT < -0.5 * T) dT = -0.5 * T;
        const double T_was = T;
        T += dT;
        if (MOMENTS ? gas::newton_done<NS>(t.m.T_mid, T_was, dT, T) : fabs(dT) <= 1e-9 * T) it_used = it + 1;
    }
    return it_used;
}

// Per-axis factors of the thread's target set (mc_target_axes).  A species' equilibrium is the energy
// set's with E = 1 and A = 0 (to the bit), so that both kinds of warp run the same code.  Returns T in
// SI.
template <int NS>
__device__ __forceinline__ double sp_target_axes(SpBlock<NS> &B, const gas::Tables &t, const UnitsF &U, double rho,
                                                 double rhoa, const double vel[3], const double vela[3], double T_lat,
                                                 AxisG<double> &G) {
    double Y;
    const double W = sp_mass_fractions(B, t, rhoa / rho, Y);
    const double T_si = si_temp(U, (float)T_lat);
    const int a = B.set < NS ? B.set : NS - 1;
    B.put(0, Y * (gas::h_RT_q(t, a, T_si) - 1.0));
    B.flip();
    if (B.set < NS) {
        const double tha = u_energy_mass(U, (float)(gas::kR * T_si / t.m.W[a]));
#pragma unroll
        for (int d = 0; d < 3; ++d) {  // axis_feq
            const double z = tha + vela[d] * vela[d];
            G.P[d][0] = 1.0 - z;
            G.P[d][1] = (vela[d] + z) * 0.5;
            G.P[d][2] = (-vela[d] + z) * 0.5;
            G.A[d][0] = G.A[d][1] = G.A[d][2] = 0.0;
        }
        G.E = 1.0;
    } else {
        const double e = u_energy_mass(U, (float)(B.sum_w(0, t) * gas::kR * T_si));
        const double theta = u_energy_mass(U, (float)(gas::kR * T_si / W));
        axis_geq(G, e, theta, vel);
    }
    return T_si;
}

// mc_state_dp with the thread's species' ratio y.
template <int NS>
__device__ __forceinline__ McDP sp_state_dp(SpBlock<NS> &B, const gas::Tables &t, const UnitsF &U, double rho_l,
                                            double p_l, double y) {
    double Y;
    const double W = sp_mass_fractions(B, t, y, Y);
    McDP s;
    const double rho_si = si_rho(U, (float)rho_l);
    const double P_si = si_p(U, (float)p_l);
    s.T = P_si * W / (rho_si * gas::kR);
    const double cpR = gas::cp_R(t, B.set < NS ? B.set : NS - 1, s.T);
    B.put(0, Y * cpR);
    B.put(1, Y * (cpR - 1.0));
    B.flip();
    const double cp = B.sum_w(0, t) * gas::kR, cv = B.sum_w(1, t) * gas::kR;
    s.c = u_u(U, (float)sqrt(cp / cv * gas::kR * s.T / W));
    s.gamma = cp / cv;
    s.Rmix = u_cp(U, (float)(gas::kR / W));
    return s;
}

// The (p, u, v, w, rho) derivatives of mc_deriv along axis d, and the thread's species' dY.
template <int NS, class AT>
__device__ __forceinline__ void sp_deriv(const AT &A, int a, long n, int d, int mode, double D[5], double &dY) {
    const long o = d == 0 ? A.si : (d == 1 ? A.sj : 1);
    const typename AT::R *R = A.rec_cur;
    const int pl[5] = {RM_P, RM_U, RM_V, RM_W, RM_RHO};
    const int pa = rs(a, RS_RHO);
    if (mode == 0) {
        const long mp = n + o, mm = n - o;
#pragma unroll
        for (int q = 0; q < 5; ++q) D[q] = (rec(A, R, pl[q], mp) - rec(A, R, pl[q], mm)) / (2.0 * 1.0);
        dY = (rec(A, R, pa, mp) / rec(A, R, RM_RHO, mp) - rec(A, R, pa, mm) / rec(A, R, RM_RHO, mm)) / (2.0 * 1.0);
        return;
    }
    const long m0 = n, m1 = mode == 1 ? n + o : n - o, m2 = mode == 1 ? n + 2 * o : n - 2 * o;
    const double k0 = mode == 1 ? -1.5 : 1.5, k1 = mode == 1 ? 2.0 : -2.0, k2 = mode == 1 ? -0.5 : 0.5;
#pragma unroll
    for (int q = 0; q < 5; ++q)
        D[q] = k0 * rec(A, R, pl[q], m0) + k1 * rec(A, R, pl[q], m1) + k2 * rec(A, R, pl[q], m2);
    dY = k0 * rec(A, R, pa, m0) / rec(A, R, RM_RHO, m0) + k1 * rec(A, R, pa, m1) / rec(A, R, RM_RHO, m1) +
         k2 * rec(A, R, pa, m2) / rec(A, R, RM_RHO, m2);
}

// mc_nscbc_outflow; `on`: the cells that have an outflow face (idir, isign), the others only
// keep the block's barriers company.
template <int NS, class AT>
__device__ __forceinline__ void sp_nscbc_outflow(SpBlock<NS> &B, const AT &A, bool on, unsigned fluid_up, long n,
                                                 int idir, int isign, double &rho_out, double &rhoa_out,
                                                 double vel_out[3], double &T_out) {
    const gas::Tables &t = *A.tab;
    const int a = B.set < NS ? B.set : NS - 1;
    const McFields c0 = mc_fields(A, n);
    const int Nax[3] = {A.Nx_glob, A.Ny, A.Nz};
    double D[3][5] = {{0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}};
    double dYn = 0.0;
    bool any_t = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int mode;
        if (d == idir) {
            mode = isign;
        } else {
            if (!(Nax[d] - 2 > 3)) continue;
            any_t = true;
            const int lo = d == 0 ? dir3(1, 0, 0) : (d == 1 ? dir3(0, 1, 0) : dir3(0, 0, 1));
            if (!((fluid_up >> lo) & 1))
                mode = 1;
            else if (d != 2 && !((fluid_up >> opp(lo)) & 1))
                mode = -1;  // the z branch of the reference tests k-1 twice, so never this case
            else
                mode = 0;
        }
        if (!on) continue;
        double dY;
        sp_deriv<NS>(A, a, n, d, mode, D[d], dY);
        if (d == idir) dYn = dY;
    }
    const double y = rec(A, A.rec_cur, rs(a, RS_RHO), n) / c0.rho;
    const McDP st = sp_state_dp(B, t, A.U, c0.rho, c0.p, y);
    const double c = st.c, rho = c0.rho, p = c0.p;
    const double u = c0.u[0], v = c0.u[1], w = c0.u[2];
    double T1 = 0.0, T5 = 0.0;
    if (any_t) {
        const double gam = st.gamma;
        if (idir == 0) {
            T1 = (v * (D[1][0] - rho * c * D[1][1])) + (w * (D[2][0] - rho * c * D[2][1])) +
                 (gam * p * (D[1][2] + D[2][3]));
            T5 = (v * (D[1][0] + rho * c * D[1][1])) + (w * (D[2][0] + rho * c * D[2][1])) +
                 (gam * p * (D[1][2] + D[2][3]));
        } else if (idir == 1) {
            T1 = (u * (D[0][0] - rho * c * D[0][2])) + (w * (D[2][0] - rho * c * D[2][2])) +
                 (gam * p * (D[0][1] + D[2][3]));
            T5 = (u * (D[0][0] + rho * c * D[0][2])) + (w * (D[2][0] + rho * c * D[2][2])) +
                 (gam * p * (D[0][1] + D[2][3]));
        } else {
            T1 = (u * (D[0][0] - rho * c * D[0][3])) + (v * (D[1][0] - rho * c * D[1][3])) +
                 (gam * p * (D[0][1] + D[1][2]));
            T5 = (u * (D[0][0] + rho * c * D[0][3])) + (v * (D[1][0] + rho * c * D[1][3])) +
                 (gam * p * (D[0][1] + D[1][2]));
        }
    }
    const double mach = sqrt(u * u + v * v + w * w) / c;
    const double un = idir == 0 ? u : (idir == 1 ? v : w);
    double Dn[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) Dn[q] = idir == 0 ? D[0][q] : (idir == 1 ? D[1][q] : D[2][q]);
    const double dp = Dn[0], dun = idir == 0 ? Dn[1] : (idir == 1 ? Dn[2] : Dn[3]), drho = Dn[4];
    double L1 = (un - c) * (dp - rho * c * dun);
    double L5 = (un + c) * (dp + rho * c * dun);
    const double Ls = un * (c * c * drho - dp);
    double Lt[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) Lt[d] = (d == idir) ? Ls : un * Dn[1 + d];
    const double L6 = un * dYn;
    const long og = idir == 0 ? A.si : (idir == 1 ? A.sj : 1);
    const double P_target = rec(A, A.rec_cur, RM_P, n - isign * og);
    const double beta = mach;
    const int Nn = idir == 0 ? Nax[0] : (idir == 1 ? Nax[1] : Nax[2]);
    if (mach < 1.0) {
        const double Kout = kNscbcSigmaOut * (1.0 - mach * mach) * (c / Nn);
        if (isign == 1)
            L5 = Kout * (p - P_target) - (1.0 - beta) * T5;
        else
            L1 = Kout * (p - P_target) - (1.0 - beta) * T1;
    }
    const double dt = A.dt;
    double dv[3];
    const double drho_t = (Ls + 0.5 * (L1 + L5)) / (c * c);
#pragma unroll
    for (int d = 0; d < 3; ++d) dv[d] = (d == idir) ? (L5 - L1) / (2.0 * c * rho) : Lt[d];
    const double dpt = 0.5 * (L1 + L5);
    rho_out = rho - dt * drho_t;
#pragma unroll
    for (int d = 0; d < 3; ++d) vel_out[d] = c0.u[d] - dt * dv[d];
    const double p_out = p - dt * dpt;
    rhoa_out = (y - dt * L6) * rho_out;
    double Y2;
    const double W2 = sp_mass_fractions(B, t, rhoa_out / rho_out, Y2);
    const double T = (double)si_p(A.U, (float)p_out) * W2 / ((double)si_rho(A.U, (float)rho_out) * gas::kR);
    T_out = u_temp(A.U, (float)T);
}

// mc_lodi_inflow for the face direction l_if of each cell.
template <int NS, class AT>
__device__ __forceinline__ void sp_lodi_inflow(SpBlock<NS> &B, const AT &A, long n, int d, int cd, double &rho_in,
                                               double &rhoa_in, double vel_in[3], double &T_in) {
    const gas::Tables &t = *A.tab;
    const int a = B.set < NS ? B.set : NS - 1, pa = rs(a, RS_RHO);
    const McFields c0 = mc_fields(A, n);
    const double ra0 = rec(A, A.rec_cur, pa, n);
    const double y = ra0 / c0.rho;
    const McDP st = sp_state_dp(B, t, A.U, c0.rho, c0.p, y);
    const double c = st.c;
    const long o = (long)cd * (d == 0 ? A.si : (d == 1 ? A.sj : 1));
    const McFields c1 = mc_fields(A, n + o), cb = mc_fields(A, n - o);
    auto pick = [](const double *v, int q) { return q == 0 ? v[0] : (q == 1 ? v[1] : v[2]); };
    const double un = pick(c0.u, d), cbn = pick(cb.u, d);
    const double dun = mc_fd_uw(un, pick(c1.u, d), cd);
    const double dp = mc_fd_uw(c0.p, c1.p, cd);
    const double dY = mc_fd_uw(y, rec(A, A.rec_cur, pa, n + o) / c1.rho, cd);
    const int Nd = d == 0 ? A.Nx_glob : (d == 1 ? A.Ny : A.Nz);
    const double rho = c0.rho;
    const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
    const double L1a = (un - c) * (dp - rho * c * dun);
    const double L2 = kLodiSigmaIn * c / Nd * rho * st.Rmix * (c0.T - cb.T);
    const double L3 = kLodiSigmaIn * c / Nd * (pick(c0.u, t1) - pick(cb.u, t1));
    const double L4 = kLodiSigmaIn * c / Nd * (pick(c0.u, t2) - pick(cb.u, t2));
    const double L5a = (un + c) * (dp + rho * c * dun);
    const double relax_K = kLodiSigmaIn * c * c / Nd * rho * (1.0 - (un / c) * (un / c));
    double L1 = L1a, L5 = L5a;
    // left boundary: the z branch of the reference tests cy here (so a z face, whose cy is 0,
    // always takes the right-boundary form)
    const bool left = (d == 2 ? 0 : cd) > 0;
    if (left)
        L5 = relax_K * (un - cbn);
    else
        L1 = relax_K * (un - cbn);
    const double d1 = 1.0 / (c * c) * (L2 + 0.5 * (L5 + L1));
    const double d2 = 1.0 / (2.0 * rho * c) * (L5 - L1);
    const double d5 = 0.5 * (L5 + L1);
    const double dt = A.dt;
    rho_in = rho - dt * d1;
    const double vn = un - dt * d2, v1 = pick(c0.u, t1) - dt * L3, v2 = pick(c0.u, t2) - dt * L4;
#pragma unroll
    for (int q = 0; q < 3; ++q) vel_in[q] = q == d ? vn : (q == t1 ? v1 : v2);
    const double p_in = c0.p - dt * d5;
    rhoa_in = (y - dt * un * dY) * rho_in;
    const double y2 = rhoa_in / rho_in;
    double Y2;
    const double W2 = sp_mass_fractions(B, t, y2, Y2);
    const double T = (double)si_p(A.U, (float)p_in) * W2 / ((double)si_rho(A.U, (float)rho_in) * gas::kR);
    T_in = u_temp(A.U, (float)T);
    const double dens = (double)si_p(A.U, (float)p_in) * W2 / (gas::kR * (double)si_temp(A.U, (float)T_in));
    rho_in = u_rho(A.U, (float)dens);
    rhoa_in = y2 * rho_in;
}

// The rest of mc_local_state, and mc_calc_temp: the cell's local state from the thread's set's
// sums s0 (density, or the energy set's rhoE) and m (momentum), and its temperature.
template <int NS, class AT>
__device__ __forceinline__ void sp_local_state(SpBlock<NS> &B, const AT &A, double s0, const double m[3], double T0_si,
                                               bool on, double &rho_loc, double vel_loc[3], double vela[3],
                                               double &T_loc) {
    const gas::Tables &t = *A.tab;
    B.put(0, s0);
#pragma unroll
    for (int d = 0; d < 3; ++d) B.put(1 + d, m[d]);
    B.flip();
    rho_loc = B.sum(0);
    const double rhoe_loc = B.get(0, NS);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        vel_loc[d] = B.sum(1 + d);
        vela[d] = s0 > 0.0 ? m[d] / s0 : 0.0;
        vel_loc[d] = rho_loc > 0 ? vel_loc[d] / rho_loc : 0.0;
    }
    B.put(0, 0.5 * s0 / rho_loc);
    B.put(1, vela[0] * vela[0] + vela[1] * vela[1] + vela[2] * vela[2]);
    B.flip();
    double Uint = rhoe_loc / rho_loc;
#pragma unroll
    for (int a = 0; a < NS; ++a) Uint = Uint - B.get(0, a) * B.get(1, a);
    // calculate_temp
    double Y, T;
    sp_mass_fractions(B, t, s0 / rho_loc, Y);
    const int it = sp_T_from_u<NS, false, false>(B, t, Y, si_energy_mass(A.U, (float)Uint), T0_si, on, T);
    if (it < 0 && B.set == 0) atomic_status(A.status, LBMGPU_ST_NEWTON);
    T_loc = u_temp(A.U, (float)T);
}

// The moments of the cell (mc_moments_cell and mc_moments_finish) from the thread's set.
template <int NS, class AT>
__device__ __forceinline__ void sp_moments(SpBlock<NS> &B, const AT &A, long n, bool valid, const double *f) {
    const gas::Tables &t = *A.tab;
    constexpr bool fast = sizeof(typename AT::P) == sizeof(float);
    const int set = B.set, lane = B.lane, a = set < NS ? set : NS - 1;
    auto &big = B.s.big;
    // the loads of the solve, before the sums
    const double T_si = si_temp(A.U, (float)rec(A, A.rec_cur, RM_T, n));
    const double p_old = rec(A, A.rec_cur, RM_P, n);
    double X_old[NS], Dr[NS];
#pragma unroll
    for (int b = 0; b < NS; ++b) {
        X_old[b] = rec(A, A.rec_cur, rs(b, RS_X), n);
        Dr[b] = b == a ? 1.0 : A.props[(long)(b < a ? pr_d<NS>(a, b) : pr_d<NS>(b, a)) * A.ncell + n];
    }
    double sums[kGsPerSpecies];
    if (set < NS) {
        species_sums(f, sums);
#pragma unroll
        for (int q = 0; q < 4; ++q) B.put(q, sums[q]);
#pragma unroll
        for (int q = 0; q < 6; ++q) big[q * NS + a][lane] = sums[4 + q];
    } else {
        double e = 0.0;
#pragma unroll
        for (int l = 0; l < 27; ++l) e += f[l];
        B.put(0, e);
    }
    B.flip();
    const double rho = B.sum(0), rhoe = B.get(0, NS);
    const double u = B.sum(1) / rho, v = B.sum(2) / rho, w = B.sum(3) / rho;
    const double ra = B.get(0, a), rho_s = ra > kSpeciesMin ? ra : kSpeciesMin;
    double P6 = 0.0;
    if (set < 6) {
#pragma unroll
        for (int b = 0; b < NS; ++b) P6 += big[set * NS + b][lane];
    }
    __syncthreads();  // the shares are read: their space takes the Stefan-Maxwell factor

    // row a of the Stefan-Maxwell matrix, its entries in the reference's order
    // (mc_stefan_maxwell; FP32 storage: mc_stefan_maxwell_fast), then the Cholesky factor column by
    // column, each thread its own row against row c
    constexpr int kDiag0 = NS * (NS - 1) / 2, kDiag = kDiag0 + NS;
    auto Lrc = [&](int r, int c) -> double & { return big[r * (r - 1) / 2 + c][lane]; };
    double Xa = 0.0;
#pragma unroll
    for (int b = 0; b < NS; ++b)
        if (b == a) Xa = X_old[b];
    double Lr[NS], d0 = rho_s == 0.0 ? 1.0 : rho_s;
    const double kf = -0.5 * (double)A.dt * p_old;
#pragma unroll
    for (int b = 0; b < NS; ++b) {
        Lr[b] = 0.0;
        if (b == a) continue;
        double m;
        if (fast)
            m = b < a ? kf * Xa * X_old[b] / Dr[b] : kf * X_old[b] * Xa / Dr[b];
        else
            m = -1.0 * (double)A.dt / 2.0 * p_old * Xa * X_old[b] / Dr[b];
        Lr[b] = m;
        d0 -= m;
    }
    if (set < NS) big[kDiag0 + a][lane] = d0;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NS; ++c) {
        double row[NS], d = big[kDiag0 + c][lane];
#pragma unroll
        for (int q = 0; q < c; ++q) {
            row[q] = Lrc(c, q);
            d -= row[q] * row[q];
        }
        const double dg = fast ? 1.0 / sqrt(d) : sqrt(d);
        if (set < NS && a > c) {
            double s = Lr[c];
#pragma unroll
            for (int q = 0; q < c; ++q) s -= Lr[q] * row[q];
            Lr[c] = fast ? s * dg : s / dg;
            Lrc(a, c) = Lr[c];
        }
        if (set == c) big[kDiag + c][lane] = dg;
        __syncthreads();
    }
    if (set < 3) {  // the two triangular solves of one axis
        double x[NS];
#pragma unroll
        for (int r = 0; r < NS; ++r) {
            double s = B.s.x[B.g ^ 1][1 + set][r][lane];
#pragma unroll
            for (int q = 0; q < r; ++q) s -= Lrc(r, q) * x[q];
            x[r] = fast ? s * big[kDiag + r][lane] : s / big[kDiag + r][lane];
        }
#pragma unroll
        for (int r = NS - 1; r >= 0; --r) {
            double s = x[r];
#pragma unroll
            for (int q = r + 1; q < NS; ++q) s -= Lrc(q, r) * x[q];
            x[r] = fast ? s * big[kDiag + r][lane] : s / big[kDiag + r][lane];
            B.s.us[set][r][lane] = x[r];
        }
    }
    __syncthreads();
    const double us[3] = {B.s.us[0][a][lane], B.s.us[1][a][lane], B.s.us[2][a][lane]};

    // temperature from the internal energy
    double Y, X, Wn;
    if (fast) {
        const double ir = 1.0 / rho;
        const double yr = rho_s * ir, yc = yr > 0.0 ? yr : 0.0;
        B.put(0, yc);
        B.flip();
        Y = yc * (1.0 / B.sum(0));
        B.put(0, Y);
        B.flip();
        Wn = 1.0 / B.sum_w(0, t);
        X = Y * t.invW[a] * Wn;
    } else {
        Wn = sp_mass_fractions(B, t, rho_s / rho, Y);
        X = Y / t.m.W[a] * Wn;
    }
    B.put(0, 0.5 * rho_s / rho);
    B.put(1, us[0] * us[0] + us[1] * us[1] + us[2] * us[2]);
    const double Ya = rho_s / rho;
    B.put(2, Ya / t.m.W[a]);
    B.put(3, Ya);
    B.flip();
    double e = rhoe / rho;
#pragma unroll
    for (int b = 0; b < NS; ++b) e = e - B.get(0, b) * B.get(1, b);
    const double gc = (double)u_cp(A.U, (float)(gas::kR * B.sum(2) / B.sum(3)));  // store_face_terms
    const double u_si = si_energy_mass(A.U, (float)e);
    const double vol = 1.0 / (double)si_rho(A.U, (float)rho);
    const double rho_n_si = 1.0 / vol;
    double Tn;
    const int it = sp_T_from_u<NS, fast, true>(B, t, Y, u_si, T_si, true, Tn);
    const double Pn = rho_n_si * gas::kR * Tn / Wn;
    const double Tl = u_temp(A.U, (float)Tn);
    if (!valid) return;

    typename AT::R *R = A.rec_nxt;
    const double um[3] = {u, v, w};
    if (set == NS) {
        put(A, R, RM_RHO, n, rho);
        put(A, R, RM_U, n, u);
        put(A, R, RM_V, n, v);
        put(A, R, RM_W, n, w);
        put(A, R, RM_T, n, Tl);
        put(A, R, RM_P, n, u_p(A.U, (float)Pn));
        put(A, R, RM_RHOE, n, rhoe);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            put(A, R, RM_QX + d, n, rho * um[d] * (1.0 - 3.0 * gc * Tl) - rho * (um[d] * um[d] * um[d]));
        if (it < 0) atomic_status(A.status, LBMGPU_ST_NEWTON);
        if (!isfinite(rho) || !isfinite(Tn) || !isfinite(u) || !isfinite(v) || !isfinite(w))
            atomic_status(A.status, LBMGPU_ST_NAN);
        else if (!(rho > 0.0) || !(Tn > 0.0))
            atomic_status(A.status, LBMGPU_ST_NEG_STATE);
        return;
    }
    if (set < 6) put(A, R, RM_P00 + set, n, P6);
    put(A, R, rs(a, RS_RHO), n, rho_s);
    put(A, R, rs(a, RS_X), n, X);
    const double Ra = t.Ra_lat[a];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        put(A, R, rs(a, RS_UX + d), n, us[d]);
        put(A, R, rs(a, RS_QX + d), n, rho_s * us[d] * (1.0 - 3.0 * Ra * Tl) - rho_s * (us[d] * us[d] * us[d]));
    }
}

// Cells blist[32 blockIdx.x ..] (32 lanes x (NS + 1) warps).  A lane past the list's end takes
// the last cell and stores nothing.
template <int NS, typename S>
__global__ void __launch_bounds__(kSpCells *(NS + 1), 1)
    k_mc_special(McArgsT<S, double> A, const long *__restrict__ blist) {
    using AT = McArgsT<S, double>;
    static_assert(NS >= 6, "the P tensor's six components are stored by the species' warps");
    __shared__ SpSmem<NS> sm;
    const int lane = threadIdx.x & 31, set = threadIdx.x >> 5;
    SpBlock<NS> B{sm, lane, set, 0};
    const gas::Tables &t = *A.tab;
    const long b0 = (long)blockIdx.x * kSpCells + lane;
    const bool valid = b0 < A.nb;
    const long b = valid ? b0 : A.nb - 1, n = blist[b];
    int i, j, k;
    cell_ijk(n, A.si, A.sj, i, j, k);
    if (set < SP_MASKS) sm.up[set][lane] = 0u;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int l = 0; l < 27; ++l) sm.dir[l] = dir_code(l);
    }
    __syncthreads();
    for (int l = set; l < 27; l += NS + 1) {
        const unsigned code = sm.dir[l];
        const int tn = mc_type_at(A, i - dec2(code & 3), j - dec2((code >> 2) & 3), k - dec2((code >> 4) & 3));
        const int kind = tn == T_O || tn == T_O_C   ? SP_OUT
                         : tn == T_I || tn == T_I_C ? SP_IN
                         : tn == T_S                ? SP_SOLID
                         : tn == T_A                ? SP_ADI
                         : tn == T_FS               ? SP_SLIP
                         : tn == T_F                ? SP_FLUID
                                                    : -1;
        if (kind >= 0) atomicOr(&sm.up[kind][lane], 1u << l);
    }
    __syncthreads();
    const unsigned out_m = sm.up[SP_OUT][lane], in_m = sm.up[SP_IN][lane], sol_m = sm.up[SP_SOLID][lane],
                   adi_m = sm.up[SP_ADI][lane], slip_m = sm.up[SP_SLIP][lane], fluid_up = sm.up[SP_FLUID][lane];
    // fluid downstream along l: fluid upstream along opp(l) (opposite directions are neighbours)
    const unsigned fluid_dn = (fluid_up & 1u) | ((fluid_up & 0x2aaaaaau) << 1) | ((fluid_up & 0x5555554u) >> 1);

    // ---- streaming (src/lbm-streaming.cpp:15-107): 27 loads of the thread's set, each from the
    // address its upstream kind asks for: kept populations along inflow and outflow directions (and
    // the energy set's along solid ones), bounce-back off solid and adiabatic cells, else the
    // upstream cell through the periodic wrap
    double f[27];
    {
        const unsigned kept_m = out_m | in_m | (set == NS ? sol_m : 0u), bounce_m = (sol_m | adi_m) & ~kept_m;
        McPull pp;
        mc_pull(A, n, pp);
        auto fetch = [&](const S *src, int plane) {
            const double v = (double)*src;
            return A.shift ? v + A.shift[plane] : v;
        };
#pragma unroll
        for (int l = 0; l < 27; ++l) {
            const bool kept = (kept_m >> l) & 1, back = (bounce_m >> l) & 1;
            const int plane = 27 * set + (back ? opp(l) : l);
            const long at = back || ((slip_m >> l) & 1) ? n : pull_idx(pp, l);
            f[l] = fetch(kept ? A.bst_cur + (long)plane * A.nb + b : A.pop_src + (long)plane * A.ncell + at, plane);
        }
        if (slip_m) {  // specular reflection (dirSlip, src/lbm-bc.cpp:1352-1399)
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
                if (!((in == 0 && A.halo_lo) || (in == A.Nx - 1 && A.halo_hi)))
                    in = ((in - 1 + (A.Nx - 2)) % (A.Nx - 2)) + 1;
                jn = ((jn - 1 + (A.Ny - 2)) % (A.Ny - 2)) + 1;
                kn = ((kn - 1 + (A.Nz - 2)) % (A.Nz - 2)) + 1;
                const int plane = 27 * set + lp;
                f[l] = fetch(A.pop_src + (long)plane * A.ncell + mc_idx(A, in, jn, kn), plane);
            }
        }
    }

    // ---- the outflow, inflow and solid passes.  A pass forms a target set (its state st_), the
    // local state of the cell with the boundary directions taken from it, and replaces
    //   outflow, solid: f by 2 f_target - f_local along boundary directions, f + f_target - f_local else;
    //   inflow: f by f_new + f_target - f_local and f + f_new - f_local, f_new the target at the local density.
    // One loop over the passes and one over the sets of factors (target, the inflow's f_new, local):
    // one copy of the code, which a block would otherwise fetch once per use.
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
        const unsigned bm = pass == 0 ? out_m : (pass == 1 ? in_m : sol_m);
        // outflow, inflow: the first direction with the type upstream and fluid downstream must be
        // a face direction (1..6); solid: any such direction
        const unsigned fm = bm & fluid_dn;
        const int li = fm ? __ffs((int)fm) - 1 : -1;
        const bool on = pass == 2 ? fm != 0 : li >= 1 && li <= 6;
        if (!__syncthreads_or(on)) continue;
        double rho_t, rhoa_t, vel_t[3], vela_t[3], T_t;
        if (pass == 2) {  // half-way interpolated target, q = 0.5
            const int a = set < NS ? set : NS - 1;
            const double q = 0.5;
#pragma unroll
            for (int d = 0; d < 3; ++d) vela_t[d] = 0.0;
            T_t = 0.0;
            // the energy set's warp forms the mixture's target, a species' warp its own velocity
            const int pu = set < NS ? rs(a, RS_UX) : (int)RM_U;
            for (unsigned mm = fm; mm; mm &= mm - 1) {
                const int l = __ffs((int)mm) - 1;
                const unsigned code = sm.dir[l];
                const long off = (long)dec2(code & 3) * A.si + (long)dec2((code >> 2) & 3) * A.sj + dec2((code >> 4) & 3);
                // a species takes the fluid side's species velocity with the solid cell's mixture
                // velocity, as the reference mixes them (src/lbm-bc.cpp:998-1000)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    vela_t[d] += (q * rec(A, A.rec_cur, pu + d, n + off) + rec(A, A.rec_cur, RM_U + d, n - off)) / (1.0 + q);
                if (set == NS)
                    T_t += (q * rec(A, A.rec_cur, RM_T, n + off) + rec(A, A.rec_cur, RM_T, n - off)) / (1.0 + q);
            }
            rhoa_t = 0.0;
            if (set < NS) {
#pragma unroll
                for (int l = 0; l < 27; ++l) rhoa_t += f[l];
            }
            const double inv = 1.0 / (on ? __popc(fm) : 1);
            B.put(0, set < NS ? rhoa_t : inv * T_t);
            B.flip();
            rho_t = B.sum(0);
            T_t = B.get(0, NS);
#pragma unroll
            for (int d = 0; d < 3; ++d) vel_t[d] = vela_t[d] = inv * vela_t[d];
        } else {
            const int d = on ? (li - 1) >> 1 : 0, sg = on ? ((li & 1) ? 1 : -1) : 1;
            if (pass == 0)
                sp_nscbc_outflow(B, A, on, fluid_up, n, d, sg, rho_t, rhoa_t, vel_t, T_t);
            else
                sp_lodi_inflow(B, A, n, d, on ? sg : 0, rho_t, rhoa_t, vel_t, T_t);
#pragma unroll
            for (int q = 0; q < 3; ++q) vela_t[q] = vel_t[q];
        }
        double rho_l = 0.0, rhoa_l = 0.0, vel_l[3], vela_l[3], T_l = 0.0;
        double rho_x = rho_t, rhoa_x = rhoa_t, vel_x[3], vela_x[3], T_x = T_t;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            vel_x[q] = vel_t[q];
            vela_x[q] = vela_t[q];
        }
#pragma unroll 1
        for (int stage = 0; stage < 3; ++stage) {
            if (stage == 1 && pass != 1) continue;
            AxisG<double> G;
            const double Tsi = sp_target_axes(B, t, A.U, rho_x, rhoa_x, vel_x, vela_x, T_x, G);
            double m[3] = {0.0, 0.0, 0.0}, s0 = 0.0;
            // e_l = B p_z + C A_z, B and C of the pair (c_x, c_y); the sums below in the reference's order
            const double r = set < NS ? rhoa_x : rho_x;
            double Bp[3][3], Cp[3][3];
#pragma unroll
            for (int ix = 0; ix < 3; ++ix) {
                const double px = r * G.P[0][ix], tx = r * (G.E * G.P[0][ix] + G.A[0][ix]);
#pragma unroll
                for (int iy = 0; iy < 3; ++iy) {
                    Bp[ix][iy] = tx * G.P[1][iy] + px * G.A[1][iy];
                    Cp[ix][iy] = px * G.P[1][iy];
                }
            }
#pragma unroll
            for (int l = 0; l < 27; ++l) {
                const int ix = cidx(cx(l)), iy = cidx(cy(l)), iz = cidx(cz(l));
                const double e = Bp[ix][iy] * G.P[2][iz] + Cp[ix][iy] * G.A[2][iz];
                const bool bd = (bm >> l) & 1;
                if (stage == 0) {
                    const double fv = bd ? e : f[l];
                    s0 += fv;
                    if (cx(l)) m[0] += fv * cx(l);
                    if (cy(l)) m[1] += fv * cy(l);
                    if (cz(l)) m[2] += fv * cz(l);
                    if (on) f[l] = pass == 1 ? fv : (bd ? 2 * e : e + f[l]);
                } else if (on) {
                    f[l] = stage == 1 ? e + f[l] : f[l] - e;
                }
            }
            if (stage == 0) {
                rhoa_l = s0;
                sp_local_state(B, A, s0, m, Tsi, on, rho_l, vel_l, vela_l, T_l);
            }
            // the next set: the inflow's f_new, or the local state
            const bool fresh = stage == 0 && pass == 1;
            rho_x = rho_l;
            rhoa_x = rhoa_l;
            T_x = fresh ? T_t : T_l;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                vel_x[q] = fresh ? vel_t[q] : vel_l[q];
                vela_x[q] = fresh ? vel_t[q] : vela_l[q];
            }
        }
    }
    // ---- moments, and the populations kept for the collision and the next streaming
    sp_moments(B, A, n, valid, f);
    if (!valid) return;
#pragma unroll
    for (int l = 0; l < 27; ++l) stpop_b(A, A.bst_nxt, 27 * set + l, b, f[l]);
}

}  // namespace lbm

namespace lbmh {

template <int NS, typename S>
int special_step(lbmgpu *h, const lbm::McArgsT<S, double> &A) {
    const unsigned blocks = (unsigned)((A.nb + lbm::kSpCells - 1) / lbm::kSpCells);
    EvPair eb{};
    ev_begin(h, K_OTHER, eb, h->side);
    lbm::k_mc_special<NS, S><<<blocks, lbm::kSpCells *(NS + 1), 0, h->side>>>(A, h->blist);
    ev_end(h, eb, h->side);
    CK(cudaGetLastError());
    return 0;
}

}  // namespace lbmh
