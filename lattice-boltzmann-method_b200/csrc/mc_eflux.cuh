// The energy-flux terms of the energy collision on the device: mc_eflux_cell (mc_cell.cuh: the per-cell
// function, with the reference's file:line references, which the host build runs), the same operations
// per value.  One thread per cell; mostly neighbour loads, so it is bound by rounds of memory latency:
// every load that does not depend on the species is issued before the cell's flag is known (at a cell
// whose neighbours exist), and the ten values of the next species are loaded while a species is
// summed.  Of the upwind mass-fraction difference only the side that is used is divided.
// Measured: 96^3 FP32 storage 209 -> 144 us (152 us at four blocks per SM), 64 x 48 x 40 FP64
// 55 -> 42 us (50 us at five blocks, which spill 120 B).
#pragma once
#include "launch.cuh"
#include "mc_cell.cuh"

namespace lbm {

template <int NS, typename S>
__global__ void __launch_bounds__(128, sizeof(S) == sizeof(float) ? 5 : 4) k_mc_eflux(McArgsT<S, double> A) {
    constexpr bool fast = sizeof(S) == sizeof(float);  // reciprocal densities and enthalpy quotients
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x, nc = A.ncell;
    if (n >= nc) return;
    lbmh::step_begin();
    const unsigned cf = A.cflag[n];
    const long m = min(max(n, A.si), nc - 1 - A.si);  // n, if it is a fluid cell
    const gas::Tables &t = *A.tab;
    const double *const Rc = A.rec_cur + m;
    auto rc = [&](int plane) { return Rc[(long)plane * nc]; };
    auto at = [&](int plane, long o) { return Rc[(long)plane * nc + o]; };
    auto prg = [&](int plane) { return A.props[(long)plane * nc + m]; };
    const long off[3] = {A.si, A.sj, 1};
    // the values of species a: density here and at the six face neighbours, velocity
    auto load = [&](int a, double (&x)[10]) {
        const int pr = rs(a, RS_RHO);
        x[0] = rc(pr);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x[1 + d] = rc(rs(a, RS_UX) + d);
            x[4 + 2 * d] = at(pr, -off[d]);
            x[5 + 2 * d] = at(pr, off[d]);
        }
    };
    double x[10];
    load(0, x);
    const double rho = rc(RM_RHO), um[3] = {rc(RM_U), rc(RM_V), rc(RM_W)}, Tl = rc(RM_T), p = rc(RM_P);
    const double om = prg(pr_omm<NS>()), om1 = prg(pr_om1<NS>()), gasconstant = prg(pr_gc<NS>());
    double rn[3][2];  // the neighbours' densities (FP32 storage: their reciprocals)
    int tl[3], th[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        rn[d][0] = at(RM_RHO, -off[d]);
        rn[d][1] = at(RM_RHO, off[d]);
        tl[d] = A.type[m - off[d]];
        th[d] = A.type[m + off[d]];
    }
    if (!(cf & CF_FLUID)) return;
    const double T_si = si_temp(A.U, (float)Tl), dt = A.dt;
    const double ir = fast ? 1.0 / rho : 0.0, invT = fast ? 1.0 / T_si : 0.0;
    if (fast) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            rn[d][0] = 1.0 / rn[d][0];
            rn[d][1] = 1.0 / rn[d][1];
        }
    }
    const double kd = om1 / (-om + om1), kc = 0.5 * (2.0 - om1) / (-om + om1) * dt * p;
    double qd[3] = {0, 0, 0}, qc[3] = {0, 0, 0};
#pragma unroll 1
    for (int a = 0; a < NS; ++a) {
        double y[10];
        load(a + 1 < NS ? a + 1 : a, y);
        const double ha =
            fast ? u_energy_mass(A.U, (float)(gas::h_RT_fast(t, a, T_si, invT) * gas::kR * T_si * t.invW[a]))
                 : u_energy_mass(A.U, (float)(gas::h_RT_q(t, a, T_si) * gas::kR * T_si / t.m.W[a]));
        const double Yc = fast ? x[0] * ir : x[0] / rho;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double du = x[1 + d] - um[d];
            qd[d] += kd * ha * x[0] * du;
            const bool lo = du > 0;  // mc_fd_fuw
            const double xn = lo ? x[4 + 2 * d] : x[5 + 2 * d], r = lo ? rn[d][0] : rn[d][1];
            const double Yn = fast ? xn * r : xn / r;
            const double dY = fuw_blocked(lo ? tl[d] : th[d]) ? 0.0 : (lo ? Yc - Yn : Yn - Yc);
            qc[d] += kc * ha * dY;
        }
#pragma unroll
        for (int q = 0; q < 10; ++q) x[q] = y[q];
    }
    double P6[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) P6[q] = rc(RM_P00 + q);
    const double Pf[3][3] = {{P6[0], P6[1], P6[2]}, {P6[1], P6[3], P6[4]}, {P6[2], P6[4], P6[5]}};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double Qc = rho * um[d] * (1.0 - 3.0 * gasconstant * Tl) - rho * (um[d] * um[d] * um[d]);
        const double dQ = mc_fd_central(at(RM_QX + d, -off[d]), Qc, at(RM_QX + d, off[d]), tl[d], th[d]);
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < 3; ++b) s += um[b] * (Pf[b][d] - ((b == d ? p : 0.0) + rho * um[b] * um[d]));
        A.props[(long)pr_dq<NS>(d) * nc + n] = s + qd[d] + qc[d] + 0.5 * dt * um[d] * dQ;
    }
}

}  // namespace lbm
