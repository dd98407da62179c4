// Streaming and moments of the interior cells (no boundary upstream) on the device, the operations of
// mc_moments_cell and mc_moments_finish (mc_cell.cuh: the per-cell functions, with the reference's
// file:line references, which the host build runs) in three kernels:
//   k_mc_gather   a block of one warp per population set and 32 cells: each thread pulls its set's 27
//                 populations and sums them; the sums over the species (density, velocity, pressure
//                 tensor) are formed from shared memory in species order, so the record's planes are
//                 written as they stay -- only the momenta j_a wait in the velocities' planes;
//   k_mc_diffuse  per cell: the Stefan-Maxwell system, j_a replaced by the species velocities;
//   k_mc_thermo   per cell: temperature, pressure, mole fractions and the face terms.
// The planes between them are the record's own (the gather wrote 91 planes of sums for the solve to
// read back; memory per cell 728 B less).  One kernel for the last two held the 9 x 9 factor and the
// temperature iteration in one thread: 255 registers, eight warps per SM, a third of the time waiting
// for memory; now three and five blocks of 128 threads per SM (168 and 96 registers; nine species spill
// 168 B in FP64 and 88 B in FP32, and 72 B).  All of a
// thread's loads are issued before its cell's flag is known.
// Measured, 96^3 FP32 storage: gather 387 -> 281 us (1456 B a cell: 4.6 TB/s), solve 456 -> 344 us;
// 48 x 40 x 37 FP64: 45 -> 44 and 108 -> 73 us.  The diffusion kernel at two blocks per SM (198
// registers): 367 for 344 us.
#pragma once
#include "launch.cuh"
#include "mc_cell.cuh"

namespace lbm {

constexpr int kGatherCells = 32;  // cells of a gather block, one per lane

// The cell of the interior nearest to n (itself for every fluid cell) and its pull: loads are issued
// there before the cell's flag is known, one round of memory latency instead of two.
template <class AT>
__device__ __forceinline__ long interior_pull(const AT &A, long n, unsigned (&X)[3], unsigned (&Y)[3], unsigned (&Z)[3]) {
    int i, j, k;
    cell_ijk(n, A.si, A.sj, i, j, k);
    i = min(max(i, 1), A.Nx - 2);
    j = min(max(j, 1), A.Ny - 2);
    k = min(max(k, 1), A.Nz - 2);
    const long m = (long)i * A.si + (long)j * A.sj + k;
    McPull pp;
    mc_pull(A, i, j, k, pp);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        X[c] = (unsigned)pp.X[c];
        Y[c] = (unsigned)pp.Y[c];
        Z[c] = (unsigned)pp.Z[c];
    }
    return m;
}

// Warps per block: one per set.
template <int NS, typename S>
__global__ void __launch_bounds__(kGatherCells *(NS + 1), sizeof(S) == sizeof(float) ? 3 : 2)
    k_mc_gather(McArgsT<S, double> A) {
    __shared__ double sm[kGsPerSpecies][NS][kGatherCells];  // the species' sums
    const int lane = threadIdx.x & 31, set = threadIdx.x >> 5;
    const long n = (long)blockIdx.x * kGatherCells + lane, nc = A.ncell;
    const bool in = n < nc;
    lbmh::step_begin();
    const unsigned cf = in ? A.cflag[n] : 0u;
    unsigned X[3], Y[3], Z[3];
    interior_pull(A, in ? n : 0, X, Y, Z);
    const S *const s0 = A.pop_src + (long)27 * set * nc;
    S v[27];
#pragma unroll
    for (int l = 0; l < 27; ++l) v[l] = (s0 + (long)l * nc)[X[cidx(cx(l))] + Y[cidx(cy(l))] + Z[cidx(cz(l))]];
    double f[27], s[kGsPerSpecies];
#pragma unroll
    for (int l = 0; l < 27; ++l) f[l] = (double)v[l];
    // FP32 storage: sums of the stored deviations plus the shift's own
    const double *const ss = A.shift + 27 * (NS + 1) + kGsPerSpecies * set;
    double *const R = A.rec_nxt;
    const bool on = cf == CF_FLUID;
    if (set < NS) {
        species_sums(f, s);
#pragma unroll
        for (int q = 0; q < kGsPerSpecies; ++q) {
            if (sizeof(S) == sizeof(float)) s[q] += ss[q];
            sm[q][set][lane] = s[q];
        }
        if (on) {
            put(A, R, rs(set, RS_RHO), n, s[0] > kSpeciesMin ? s[0] : kSpeciesMin);
#pragma unroll
            for (int d = 0; d < 3; ++d) put(A, R, rs(set, RS_UX + d), n, s[1 + d]);
        }
    } else {
        double e = sizeof(S) == sizeof(float) ? ss[0] : 0.0;
#pragma unroll
        for (int l = 0; l < 27; ++l) e += f[l];
        if (on) put(A, R, RM_RHOE, n, e);
    }
    __syncthreads();
    if (!on) return;
    auto total = [&](int q) {
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < NS; ++a) v += sm[q][a][lane];
        return v;
    };
    for (int task = set; task < 10; task += NS + 1) {
        if (task < 6) {
            put(A, R, RM_P00 + task, n, total(4 + task));
        } else {
            const double rho = total(0);
            put(A, R, task == 6 ? RM_RHO : RM_U + task - 7, n, task == 6 ? rho : total(task - 6) / rho);
        }
    }
}

// The Stefan-Maxwell system of every interior cell (mc_stefan_maxwell, in FP32 storage the reciprocal
// forms of mc_stefan_maxwell_fast) with the D_ab the collision of this step evaluated.
template <int NS, typename S>
__global__ void __launch_bounds__(128, 3) k_mc_diffuse(McArgsT<S, double> A) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= A.ncell) return;
    lbmh::step_begin();
    const unsigned cf = A.cflag[n];
    // every load before the flag is known
    double *const R = A.rec_nxt;
    double L[NS][NS], X[NS], rho_s[NS], j[NS][3], us[NS][3];  // L: lower triangle and diagonal only
#pragma unroll
    for (int a = 0; a < NS; ++a)
#pragma unroll
        for (int b = 0; b < a; ++b) L[a][b] = A.props[(long)pr_d<NS>(a, b) * A.ncell + n];
    const double p_old = rec(A, A.rec_cur, RM_P, n);
#pragma unroll
    for (int a = 0; a < NS; ++a) {
        X[a] = rec(A, A.rec_cur, rs(a, RS_X), n);
        rho_s[a] = rec(A, R, rs(a, RS_RHO), n);
#pragma unroll
        for (int d = 0; d < 3; ++d) j[a][d] = rec(A, R, rs(a, RS_UX + d), n);
    }
    if (cf != CF_FLUID) return;
    if constexpr (sizeof(S) == sizeof(float))
        mc_stefan_maxwell_fast<NS>(A.dt, p_old, X, rho_s, j, L, us);
    else
        mc_stefan_maxwell<NS, double>(A.dt, p_old, X, rho_s, j, L, us);
#pragma unroll
    for (int a = 0; a < NS; ++a)
#pragma unroll
        for (int d = 0; d < 3; ++d) put(A, R, rs(a, RS_UX + d), n, us[a][d]);
}

// Temperature from the internal energy (setState_UV, lbm-moment.cpp:346-368), pressure, mole
// fractions and the face terms of every interior cell.
template <int NS, typename S>
__global__ void __launch_bounds__(128, 5) k_mc_thermo(McArgsT<S, double> A) {
    constexpr bool fast = sizeof(S) == sizeof(float);
    __shared__ gas::ThermoTab<NS> tab;  // the temperature iteration's coefficients
    const gas::Tables &t = *A.tab;
    tab.fill(t, threadIdx.x, blockDim.x);
    __syncthreads();
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= A.ncell) return;
    lbmh::step_begin();
    const unsigned cf = A.cflag[n];
    double *const R = A.rec_nxt;
    const double rho = rec(A, R, RM_RHO, n), rhoe = rec(A, R, RM_RHOE, n);
    const double um[3] = {rec(A, R, RM_U, n), rec(A, R, RM_V, n), rec(A, R, RM_W, n)};
    const double T_si = si_temp(A.U, (float)rec(A, A.rec_cur, RM_T, n));
    double Yr[NS], v2[NS];  // rho_a / rho, |u_a|^2
#pragma unroll
    for (int a = 0; a < NS; ++a) {
        Yr[a] = rec(A, R, rs(a, RS_RHO), n);
        const double u = rec(A, R, rs(a, RS_UX), n), v = rec(A, R, rs(a, RS_UX + 1), n), w = rec(A, R, rs(a, RS_UX + 2), n);
        v2[a] = u * u + v * v + w * w;
    }
    if (cf != CF_FLUID) return;
    const double ir = fast ? 1.0 / rho : 0.0;
    double Y[NS], Wn, gc, e = rhoe / rho;
    {
        double X[NS], sYW = 0.0, sY = 0.0;  // the composition gas constant of store_face_terms
#pragma unroll
        for (int a = 0; a < NS; ++a) {
            Yr[a] = fast ? Yr[a] * ir : Yr[a] / rho;
            sYW += fast ? Yr[a] * t.invW[a] : Yr[a] / t.m.W[a];
            sY += Yr[a];
        }
        gc = (double)u_cp(A.U, (float)(gas::kR * sYW / sY));
        Wn = fast ? set_mass_fractions_fast<NS>(t, Yr, Y, X) : set_mass_fractions<NS>(t, Yr, Y, X);
#pragma unroll
        for (int a = 0; a < NS; ++a) {
            e = e - 0.5 * Yr[a] * v2[a];
            put(A, R, rs(a, RS_X), n, X[a]);
        }
    }
    const double u_si = si_energy_mass(A.U, (float)e);
    const double vol = 1.0 / (double)si_rho(A.U, (float)rho);
    const double rho_n_si = 1.0 / vol;
    double Tn;
    if (gas::T_from_u_tab<NS, fast>(tab, Y, u_si, T_si, Tn) < 0) atomic_status(A.status, LBMGPU_ST_NEWTON);
    const double Pn = rho_n_si * gas::kR * Tn / Wn;
    const double Tl = u_temp(A.U, (float)Tn);
    put(A, R, RM_T, n, Tl);
    put(A, R, RM_P, n, u_p(A.U, (float)Pn));
    // the face terms (store_face_terms), the species' values read again rather than held in registers
#pragma unroll
    for (int d = 0; d < 3; ++d)
        put(A, R, RM_QX + d, n, rho * um[d] * (1.0 - 3.0 * gc * Tl) - rho * (um[d] * um[d] * um[d]));
#pragma unroll
    for (int a = 0; a < NS; ++a) {
        const double ra = rec(A, R, rs(a, RS_RHO), n), k = 1.0 - 3.0 * t.Ra_lat[a] * Tl;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double u = rec(A, R, rs(a, RS_UX + d), n);
            put(A, R, rs(a, RS_QX + d), n, ra * u * k - ra * (u * u * u));
        }
    }
    if (!isfinite(rho) || !isfinite(Tn) || !isfinite(um[0]) || !isfinite(um[1]) || !isfinite(um[2]))
        atomic_status(A.status, LBMGPU_ST_NAN);
    else if (!(rho > 0.0) || !(Tn > 0.0))
        atomic_status(A.status, LBMGPU_ST_NEG_STATE);
}

}  // namespace lbm
