// Single-component thermal D3Q27 step kernels (the reference with MULTICOMP off).
//
// Device state (structure of arrays; cell index n = (i*Ny + j)*Nz + k, k fastest, ghosts
// included so the neighbour arithmetic is the reference's):
//   pop[2] : 54 planes of ncell doubles -- f directions 0..26, then g directions 0..26.
//            The post-collision populations fpc/gpc of the last step, or -- right after an
//            upload or Init ("local" mode) -- the populations f/g themselves.
//   mom[2] : M_N planes -- the per-cell record the collision and the neighbours read:
//            rho, u, v, w, T, p; the face-difference term Q_a = rho u_a (1 - 3 R T) - rho u_a^3
//            for a = x, y, z (src/lbm-collision.cpp:65-67); and the two collision inputs
//            that need the full pressure tensor and rho*E:
//              S_b = sum_a u_a (P_ab - P^eq_ab)   (src/lbm-collision.cpp:72-74 without the FD part)
//              Uint = rhoE/rho - |u|^2/2         (src/lbm-collision.cpp:40)
//            Double-buffered: the boundary step of step n+1 reads step n's record while
//            the moment step writes step n+1's.
//   bst[2] : 54 values per "special" cell (a fluid cell with a solid, adiabatic, free-slip,
//            inflow or outflow neighbour upstream): its post-boundary populations f, g.
//            Populations along inflow/outflow (f and g) and solid (g) directions persist
//            from step to step in the reference (src/lbm-streaming.cpp:25-32, 63-87).
//
// One time step = k_sc_collide (pop[cur] -> pop[nxt]) + k_sc_stream_moment and k_sc_special
// (sc_special.cuh; pull pop[nxt], boundary treatment, moments -> mom[nxt], bst[nxt]); then
// cur <-> nxt.
#pragma once
#include <cstdint>
#include "d3q27.cuh"

namespace lbm {

enum : int {
    M_RHO = 0, M_U = 1, M_V = 2, M_W = 3, M_T = 4, M_P = 5, M_QX = 6, M_QY = 7, M_QZ = 8,
    M_SX = 9, M_SY = 10, M_SZ = 11, M_UINT = 12, M_N = 13
};

struct ScGeom {
    int Nx, Ny, Nz;
    long ncell;
    long sj, si;  // strides of j and i (Nz, Ny*Nz)
};

struct ScPhys {
    double nu, R, gamma, prtl, dt, cv, cp;
};

__device__ __forceinline__ void raise_status(unsigned *flags, unsigned bits) { atomicOr(flags, bits); }

__device__ __forceinline__ long nb_index(const ScGeom &g, long n, int dx, int dy, int dz) {
    return n + dx * g.si + dy * g.sj + dz;
}

__device__ __forceinline__ int type_at(const ScGeom &g, const int8_t *__restrict__ type, int i, int j, int k) {
    return type[(long)i * g.si + (long)j * g.sj + k];
}

// Source-cell offsets of the pull for a cell none of whose upstream neighbours is a
// boundary cell: per axis, the upstream coordinate for c = 0, +1, -1 with the reference's
// periodic wrap (a neighbour index of 0 maps to N-2, N-1 maps to 1;
// src/lbm-streaming.cpp:101-105).  The 27 source cells are then sums of one entry per axis,
// with no branch and no type lookup.
struct PullSrc {
    int X[3], Y[3], Z[3];  // cell offsets (a single-component lattice has < 2^31 cells)
};

__device__ __forceinline__ void pull_src(const ScGeom &g, int i, int j, int k, PullSrc &s) {
    const int im = (i - 1 == 0) ? g.Nx - 2 : i - 1, ip = (i + 1 == g.Nx - 1) ? 1 : i + 1;
    const int jm = (j - 1 == 0) ? g.Ny - 2 : j - 1, jp = (j + 1 == g.Ny - 1) ? 1 : j + 1;
    const int km = (k - 1 == 0) ? g.Nz - 2 : k - 1, kp = (k + 1 == g.Nz - 1) ? 1 : k + 1;
    s.X[0] = i * (int)g.si;
    s.X[1] = im * (int)g.si;
    s.X[2] = ip * (int)g.si;
    s.Y[0] = j * (int)g.sj;
    s.Y[1] = jm * (int)g.sj;
    s.Y[2] = jp * (int)g.sj;
    s.Z[0] = k;
    s.Z[1] = km;
    s.Z[2] = kp;
}

__device__ __forceinline__ void pull_src(const ScGeom &g, long n, PullSrc &s) {
    int i, j, k;
    cell_ijk(n, g.si, g.sj, i, j, k);
    pull_src(g, i, j, k, s);
}
// The pull of the interior cell nearest to n (returned; n itself for every fluid cell), so that loads
// can be issued before the cell's flag is known.
__device__ __forceinline__ long pull_interior(const ScGeom &g, long n, PullSrc &s) {
    int i, j, k;
    cell_ijk(n, g.si, g.sj, i, j, k);
    i = min(max(i, 1), g.Nx - 2);
    j = min(max(j, 1), g.Ny - 2);
    k = min(max(k, 1), g.Nz - 2);
    pull_src(g, i, j, k, s);
    return (long)i * g.si + (long)j * g.sj + k;
}

__device__ __forceinline__ int pull_at(const PullSrc &s, int l) {
    return s.X[cidx(cx(l))] + s.Y[cidx(cy(l))] + s.Z[cidx(cz(l))];
}

// The per-axis factors with u_a^2 rounded by itself before theta is added, for the axes from FIRST on; the
// axes before are left to the compiler, which fuses a product with one use only into the sum.  With
// CUDA 12.9 both population sets, in their own threads, and the steps after an upload and later ones then
// round as they did in one thread per cell, to the bit; another compiler's choice, or one rounding for all
// axes, is as good a rounding (1e-12 of each field's scale), but a velocity component that has
// decayed to 1e-7 of the sound speed moves by 1e-9 of itself with it.
template <int FIRST>
__device__ __forceinline__ void axis_feq_sc(AxisF<double> &F, const double u[3], double theta, const double corr[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double z = theta + (a < FIRST ? u[a] * u[a] : __dmul_rn(u[a], u[a])) + corr[a];
        F.v[a][0] = 1.0 - z;
        F.v[a][1] = (u[a] + z) * 0.5;
        F.v[a][2] = (-u[a] + z) * 0.5;
    }
}
template <int FIRST>
__device__ __forceinline__ void axis_geq_sc(AxisG<double> &G, double U, double theta, const double u[3]) {
    axis_geq(G, U, theta, u);
#pragma unroll
    for (int a = FIRST; a < 3; ++a) {
        const double z = theta + __dmul_rn(u[a], u[a]);
        G.P[a][0] = 1.0 - z;
        G.P[a][1] = (u[a] + z) * 0.5;
        G.P[a][2] = (-u[a] + z) * 0.5;
    }
}

// Sums of the moments of one cell: rho, j, P (upper triangle), rhoe, q.
struct ScSums {
    double rho, j[3], P[6], re, q[3];
};

__device__ __forceinline__ void sums_init(ScSums &s) {
    s.rho = 0;
    s.re = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        s.j[a] = 0;
        s.q[a] = 0;
    }
#pragma unroll
    for (int a = 0; a < 6; ++a) s.P[a] = 0;
}

// Adds direction l's populations (in the reference's summation order, lbm-moment.cpp:35-53).
__device__ __forceinline__ void sums_add(ScSums &s, int l, double fv, double gv) {
    s.rho += fv;
    if (cx(l)) s.j[0] += cx(l) * fv;
    if (cy(l)) s.j[1] += cy(l) * fv;
    if (cz(l)) s.j[2] += cz(l) * fv;
    if (cx(l)) s.P[0] += fv;
    if (cx(l) * cy(l)) s.P[1] += cx(l) * cy(l) * fv;
    if (cx(l) * cz(l)) s.P[2] += cx(l) * cz(l) * fv;
    if (cy(l)) s.P[3] += fv;
    if (cy(l) * cz(l)) s.P[4] += cy(l) * cz(l) * fv;
    if (cz(l)) s.P[5] += fv;
    s.re += gv;
    if (cx(l)) s.q[0] += cx(l) * gv;
    if (cy(l)) s.q[1] += cy(l) * gv;
    if (cz(l)) s.q[2] += cz(l) * gv;
}

// The face-difference quantity of the collision's FD correction (src/lbm-collision.cpp:65-67).
__device__ __forceinline__ double qdev(double rho, double ua, double T, double R) {
    return rho * ua * (1.0 - 3.0 * R * T) - rho * (ua * ua * ua);
}

// The collision inputs that need the full pressure tensor and rho*E
// (src/lbm-collision.cpp:40-54, 72-74): S_b = sum_a u_a (P_ab - (p delta_ab + rho u_a u_b)),
// Uint = rhoE/rho - |u|^2/2.
__device__ __forceinline__ void coll_inputs(double rho, const double u[3], double p, const double P6[6], double rhoe,
                                            double S[3], double &Uint) {
    const double Pf[3][3] = {{P6[0], P6[1], P6[2]}, {P6[1], P6[3], P6[4]}, {P6[2], P6[4], P6[5]}};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        double s = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) s += u[a] * (Pf[a][b] - ((a == b ? p : 0.0) + rho * u[a] * u[b]));
        S[b] = s;
    }
    Uint = rhoe / rho - 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
}

// Stores the step record of a fluid cell from its post-stream moment sums (reference
// LBM::calculate_moment, src/lbm-moment.cpp:11-125), with the state checks.
__device__ __forceinline__ void store_record_sc(const ScGeom &g, const ScPhys &P, long n, const ScSums &s,
                                                double *__restrict__ mom, unsigned *status) {
    const long nc = g.ncell;
    const double rho = s.rho;
    const double u[3] = {s.j[0] / rho, s.j[1] / rho, s.j[2] / rho};
    const double Uint0 = s.re / rho - 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    const double T = Uint0 / P.cv;
    const double p = rho * P.R * T;
    double S[3], Uint;
    coll_inputs(rho, u, p, s.P, s.re, S, Uint);
    mom[M_RHO * nc + n] = rho;
    mom[M_U * nc + n] = u[0];
    mom[M_V * nc + n] = u[1];
    mom[M_W * nc + n] = u[2];
    mom[M_T * nc + n] = T;
    mom[M_P * nc + n] = p;
    mom[M_QX * nc + n] = qdev(rho, u[0], T, P.R);
    mom[M_QY * nc + n] = qdev(rho, u[1], T, P.R);
    mom[M_QZ * nc + n] = qdev(rho, u[2], T, P.R);
    mom[M_SX * nc + n] = S[0];
    mom[M_SY * nc + n] = S[1];
    mom[M_SZ * nc + n] = S[2];
    mom[M_UINT * nc + n] = Uint;
    if (!isfinite(rho) || !isfinite(T) || !isfinite(u[0]) || !isfinite(u[1]) || !isfinite(u[2]))
        raise_status(status, LBMGPU_ST_NAN);
    else if (!(rho > 0.0) || !(T > 0.0))
        raise_status(status, LBMGPU_ST_NEG_STATE);
}

}  // namespace lbm
