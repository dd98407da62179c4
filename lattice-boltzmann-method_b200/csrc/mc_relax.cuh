// The population update of the multicomponent collision on the device: mc_relax_species and
// mc_relax_energy (mc_cell.cuh: the per-cell functions, with the reference's file:line references,
// which the host build runs) with the arithmetic arranged for the instruction count.
//
// One thread per (cell, population set): blockIdx.y = set, so a warp reads one set's planes at
// 32 consecutive cells.  Per thread 27 populations in, 27 out, some 20 record and parameter values.
// The kernel is bound by instructions and by rounds of memory latency (16 warps per SM at 128
// registers), not by HBM alone, so
//   * all loads are issued before the cell's flag is known (interior_pull): one round instead of two
//     (96^3, FP32 storage, stiff chemistry: 975 -> 838 us; without effect in FP64);
//   * a vanishing species (rho_a at the reference's floor: six of nine in a mixing layer) is copied
//     without pulling, or with chemistry takes its old populations in one batch of loads instead
//     of one per direction (838 -> 712 us; without chemistry, 96 x 80 x 72: 638 -> 343 us FP32,
//     733 -> 495 us FP64);
//   * the 27 pulls use one 64-bit base per plane, uniform over the block, and a 32-bit offset (a
//     set's 27 planes hold fewer than 2^32 values: a lattice of more cells would not fit the device);
//   * the equilibria run in the order of their factors, a pair (c_x, c_y) formed once for its three
//     directions, and in FP32 storage the stored deviations are relaxed as they are (1722 -> 1236
//     instructions per thread; 1118 -> 975 us);
//   * chemistry (the f_r term and its loads) is a template parameter.
// The next cells' values copied into shared memory meanwhile (cp.async, eight chunks of cells per
// block) was slower: 1086 us for 975, FP64 178 us for 104 at 48 x 40 x 37 -- the copies of 4 and 8
// bytes cost more issue slots than the latency they hide.
#pragma once
#include "launch.cuh"
#include "mc_cell.cuh"
#include "mc_moments.cuh"

namespace lbm {

// Blocks of 128 threads per SM (128 registers; with chemistry 216 B of spills in FP64, 96 B in FP32,
// without it none).  Five (96 registers) spill 340 B: 971 for 975 us in FP32, 111 for
// 104 us in FP64.
constexpr int kRelaxBlocks = 4;

// The 27 stored populations of set a: pulled to interior cell m, or (local mode) in place.
template <class AT>
__device__ __forceinline__ void relax_fetch(const AT &A, long m, int a, const unsigned (&X)[3], const unsigned (&Y)[3],
                                            const unsigned (&Z)[3], typename AT::P (&v)[27]) {
    const typename AT::P *const s0 = A.pop_src + (long)27 * a * A.ncell;
    if (A.local) {
#pragma unroll
        for (int l = 0; l < 27; ++l) v[l] = (s0 + (long)l * A.ncell)[(unsigned)m];
    } else {
#pragma unroll
        for (int l = 0; l < 27; ++l)
            v[l] = (s0 + (long)l * A.ncell)[X[cidx(cx(l))] + Y[cidx(cy(l))] + Z[cidx(cz(l))]];
    }
}
// ... and of a cell with a boundary upstream: from the boundary store.
template <class AT>
__device__ __forceinline__ void relax_fetch_special(const AT &A, long n, int a, typename AT::P (&v)[27]) {
    const typename AT::P *const s0 = A.bst_cur + A.bid[n] + (long)27 * a * A.nb;
#pragma unroll
    for (int l = 0; l < 27; ++l) v[l] = s0[l * A.nb];
}

// BGK update of species a at cell n (lbm-collision.cpp:446-519).  FP32 storage: the populations stay
// the deviations they are stored as -- their momentum plus the shift's own (ssum), each equilibrium
// against the shift of its plane (sh) -- so a thread holds 27 floats.
template <int NS, bool CHEM, class AT>
__device__ __forceinline__ void relax_species_dev(const AT &A, long n, bool in, int a, const double *sh,
                                                  const double *ssum) {
    using P = typename AT::P;
    constexpr bool shifted = sizeof(P) == sizeof(float);
    const long nc = A.ncell;
    const double *const Rc = A.rec_cur, *const Pr = A.props;
    P *const dst = A.pop_dst + (long)27 * a * nc;
    const P *const prev = A.pop_prev + (long)27 * a * nc;
    // every load before the first use, at the interior cell m (n, if it is a fluid cell)
    const unsigned cf = in ? A.cflag[n] : 0u;
    unsigned X[3], Y[3], Z[3];
    const long m = interior_pull(A, in ? n : 0, X, Y, Z);
    const double *const Ra = Rc + (long)rs(a, 0) * nc + m;
    const double rho_a = Ra[RS_RHO * nc];
    // a vanishing species keeps the old populations, except along directions where chemistry adds
    const bool low = rho_a <= kSpeciesMin;
    if (!CHEM && shifted) __syncthreads();  // the shifts are in shared memory
    if (!CHEM && low) {  // known before its populations are pulled: copied in place
        if (!(cf & CF_FLUID) || A.local) return;
        P w[27];
#pragma unroll
        for (int l = 0; l < 27; ++l) w[l] = prev[(long)l * nc + n];
#pragma unroll
        for (int l = 0; l < 27; ++l) dst[(long)l * nc + n] = w[l];
        return;
    }
    P v[27];
    relax_fetch(A, m, a, X, Y, Z, v);
    const double Tl = Rc[RM_T * nc + m], om = Pr[(long)pr_om<NS>(a) * nc + m];
    double q[3][3], fsh[3], um[3] = {0.0, 0.0, 0.0}, drho = 0.0;
    int tl[3], th[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long off = d == 0 ? A.si : (d == 1 ? A.sj : 1);
        const double *const pq = Ra + (long)(RS_QX + d) * nc;
        q[d][0] = *(pq - off);
        q[d][1] = *pq;
        q[d][2] = pq[off];
        tl[d] = A.type[m - off];
        th[d] = A.type[m + off];
        fsh[d] = Pr[(long)pr_f<NS>(a, d) * nc + m];
        if (CHEM) um[d] = Rc[(RM_U + d) * nc + m];
    }
    if (CHEM) drho = Pr[(long)pr_drho<NS>(a) * nc + m];
    if (CHEM && shifted) __syncthreads();  // the shifts are in shared memory
    if (!(cf & CF_FLUID)) return;
    if ((cf & CF_SPECIAL) && !A.local) relax_fetch_special(A, n, a, v);
    // bare species velocity sum f c / rho_a (lbm-collision.cpp:446-454)
    double ux[3] = {0.0, 0.0, 0.0};
    if (shifted) {
#pragma unroll
        for (int d = 0; d < 3; ++d) ux[d] = ssum[d];
    }
#pragma unroll
    for (int l = 0; l < 27; ++l) {
        const double f = (double)v[l];
        if (cx(l)) ux[0] += f * cx(l);
        if (cy(l)) ux[1] += f * cy(l);
        if (cz(l)) ux[2] += f * cz(l);
    }
    // the floats again below, not the doubles just made of them: those would take 54 registers
    if constexpr (shifted) {
#pragma unroll
        for (int l = 0; l < 27; ++l) asm volatile("" : "+f"(v[l]));
    }
    const double theta = A.tab->Ra_lat[a] * Tl, kc = A.dt * (2.0 - om) / (2.0 * rho_a * om);
    double corr[3], udu[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {  // FD of the face terms the moment kernels stored (lbm-collision.cpp:487-497)
        ux[d] = ux[d] / rho_a;
        corr[d] = kc * mc_fd_central(q[d][0], q[d][1], q[d][2], tl[d], th[d]);
        udu[d] = ux[d] + fsh[d];
    }
    AxisF<double> Fe, Fd, Fr;
    axis_feq(Fe, ux, theta, corr);
    axis_feq(Fd, udu, theta, corr);
    const double zero[3] = {0.0, 0.0, 0.0};
    if (CHEM) axis_feq(Fr, um, theta, zero);
    // f(l, f_e, f_d, f_r) for every direction
    auto directions = [&](const auto &f) {
#pragma unroll
        for (int ix = 0; ix < 3; ++ix) {
            const double ex = rho_a * Fe.v[0][ix], dx = rho_a * Fd.v[0][ix], rx = CHEM ? drho * Fr.v[0][ix] : 0.0;
#pragma unroll
            for (int iy = 0; iy < 3; ++iy) {
                const double ey = ex * Fe.v[1][iy], dy = dx * Fd.v[1][iy], ry = CHEM ? rx * Fr.v[1][iy] : 0.0;
#pragma unroll
                for (int iz = 0; iz < 3; ++iz)
                    f(dir3(ix, iy, iz), ey * Fe.v[2][iz], dy * Fd.v[2][iz], CHEM ? ry * Fr.v[2][iz] : 0.0);
            }
        }
    };
    auto update = [&](int l, double fe, double fd, double fr) {
        const double f = (double)v[l];
        const double out = f + om * ((shifted ? fe - sh[l] : fe) - f) + (fd - fe);
        return (P)(CHEM ? out + fr : out);
    };
    if (!CHEM || !low) {
        directions([&](int l, double fe, double fd, double fr) { dst[(long)l * nc + n] = update(l, fe, fd, fr); });
    } else if (!A.local) {
        P w[27];
#pragma unroll
        for (int l = 0; l < 27; ++l) w[l] = prev[(long)l * nc + n];
        directions([&](int l, double fe, double fd, double fr) {
            dst[(long)l * nc + n] = fr <= 0.0 ? w[l] : update(l, fe, fd, fr);
        });
    } else {
        directions([&](int l, double fe, double fd, double fr) {
            if (!(fr <= 0.0)) dst[(long)l * nc + n] = update(l, fe, fd, fr);
        });
    }
}

// Update of the energy populations at cell n (lbm-collision.cpp:317-324); the energy equilibrium's
// four products regrouped per direction as B p_z + C A_z, with B = rho ((E p_x + A_x) p_y + p_x A_y)
// and C = rho p_x p_y of its (c_x, c_y) pair.
template <int NS, class AT>
__device__ __forceinline__ void relax_energy_dev(const AT &A, long n, bool in, const double *sh) {
    using P = typename AT::P;
    constexpr bool shifted = sizeof(P) == sizeof(float);
    const long nc = A.ncell;
    const double *const Rc = A.rec_cur, *const Pr = A.props;
    const unsigned cf = in ? A.cflag[n] : 0u;
    unsigned X[3], Y[3], Z[3];
    const long m = interior_pull(A, in ? n : 0, X, Y, Z);
    P v[27];
    relax_fetch(A, m, NS, X, Y, Z, v);
    auto prg = [&](int plane) { return Pr[(long)plane * nc + m]; };
    const double rho = Rc[RM_RHO * nc + m];
    const double um[3] = {Rc[RM_U * nc + m], Rc[RM_V * nc + m], Rc[RM_W * nc + m]};
    const double om = prg(pr_omm<NS>()), om1 = prg(pr_om1<NS>());
    const double dq[3] = {prg(pr_dq<NS>(0)), prg(pr_dq<NS>(1)), prg(pr_dq<NS>(2))};
    const double Ui = prg(pr_uint<NS>()), theta = prg(pr_theta<NS>());
    if (shifted) __syncthreads();  // the shifts are in shared memory
    if (!(cf & CF_FLUID)) return;
    if ((cf & CF_SPECIAL) && !A.local) relax_fetch_special(A, n, NS, v);
    AxisG<double> G;
    axis_geq(G, Ui, theta, um);
    P *const dst = A.pop_dst + (long)27 * NS * nc;
    // the flux correction acts along the six axes; a value of it that is not finite reaches what the products
    // with zero reach in the reference: the other axes (kq), and every direction (omn)
    const double omn = om1 + 0.0 * (om1 - om), kq = 0.5 * (om1 - om) + 0.0 * dq[0] + 0.0 * dq[1] + 0.0 * dq[2];
#pragma unroll
    for (int ix = 0; ix < 3; ++ix) {
        const double px = rho * G.P[0][ix], tx = rho * (G.E * G.P[0][ix] + G.A[0][ix]);
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            const double B = tx * G.P[1][iy] + px * G.A[1][iy], C = px * G.P[1][iy];
#pragma unroll
            for (int iz = 0; iz < 3; ++iz) {
                const int l = dir3(ix, iy, iz);
                const double g = (double)v[l], gq = B * G.P[2][iz] + C * G.A[2][iz];
                double out = g + omn * ((shifted ? gq - sh[l] : gq) - g);
                if (csq(l) == 1) out += kq * (cx(l) ? cx(l) * dq[0] : (cy(l) ? cy(l) * dq[1] : cz(l) * dq[2]));
                dst[(long)l * nc + n] = (P)out;
            }
        }
    }
}

template <int NS, bool CHEM, typename S>
__global__ void __launch_bounds__(128, kRelaxBlocks) k_mc_relax(McArgsT<S, double> A) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int a = blockIdx.y;
    lbmh::step_begin();
    __shared__ double sh[30];  // FP32 storage: the set's 27 shifts and their momentum
    if (sizeof(S) == sizeof(float) && threadIdx.x < 30)
        sh[threadIdx.x] = A.shift[threadIdx.x < 27 ? 27 * a + threadIdx.x : 27 * (NS + 1) + kGsPerSpecies * a + 1 + threadIdx.x - 27];
    if (a < NS)
        relax_species_dev<NS, CHEM>(A, n, n < A.ncell, a, sh, sh + 27);
    else
        relax_energy_dev<NS>(A, n, n < A.ncell, sh);
}

}  // namespace lbm
