// lbmgpu, multicomponent path: the chemistry's kernels and their launches, for one species count
// NS, in a compilation unit of their own (mc_chem<NS>.cu): LBMGPU_CHEM_ROSENBROCK (ROS2 of every
// cell, the surrogate's use, the integrator list) and LBMGPU_CHEM_REF_EXPLICIT.  They read the
// record and write the chemistry's collision parameters, no populations; the stiff chemistry's
// arithmetic does not depend on the population storage either, so one instance serves both.
#pragma once
#include <type_traits>

#include "handle.cuh"
#include "mc_cell.cuh"
#include "mc_ops.cuh"

namespace {

using namespace lbm;
using namespace lbmh;

// The cells the surrogate leaves to the integrator (sur.ilist), G lanes per cell: the
// lanes of a group evaluate the finite-difference Jacobian's columns side by side
// (gas::ros2_advance_group), so the listed cells do not wait on serial integrations of one
// lane each.  A short list (up to kChemShortList cells: latency-bound) takes 8 lanes per
// cell, a long one 4 (the group's redundant factorisation then costs more than the
// latency it saves); the choice is made on the device from the list's length.
// The stiff integrator's iteration matrix in shared memory, m^2 doubles per thread of a block
// (kernels over a compiled mechanism; m the unknowns of its iteration system, gas::SysMap: 9
// for the H2/air mechanism, whose N2 is inert): two blocks of 128 threads per SM hold 162 kB,
// where the thread's own array would live in local memory (its pivoted rows are indexed at
// run time) and spill through L2; what the blocks leave of the SM's 256 kB serves as L1.
constexpr bool kChemSharedMat = true;
template <int NS, class KIN>
constexpr size_t chem_smem_bytes() {
    constexpr size_t m = gas::SysMap<KIN, NS + 1>::size;
    return kChemSharedMat ? m * m * kBlock * sizeof(double) : 0;
}
constexpr unsigned kChemShortList = 5000;
template <int NS, int G, class KIN, bool SMAT = false>
__device__ __forceinline__ void chem_list_groups(const McArgs &A, unsigned cnt) {
    const unsigned groups = gridDim.x * blockDim.x / G;
    for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) / G; i < cnt; i += groups) {
        const long n = A.sur.ilist[i];
        double rho, rho_a[NS], Y[NS], T_si, rho_si, P_si;
        mc_chem_state<NS>(A, n, rho, rho_a, Y, T_si, rho_si, P_si);
        mc_chem_ros2<NS, McArgs, true, G, KIN, SMAT>(A, n, rho, rho_a, Y, T_si, rho_si, P_si, false);
    }
}
// With a compiled mechanism (KIN: analytic species Jacobian, two right-hand sides per
// sub-step besides it) a cell is one lane's work, its iteration matrix in shared memory as in
// k_mc_chem (launched with chem_smem_bytes).
template <int NS, class KIN = void>
__global__ void __launch_bounds__(kBlock, 2) k_mc_chem_list(McArgs A) {
    const unsigned cnt = *A.sur.icount;
    if constexpr (!std::is_void_v<KIN>)
        chem_list_groups<NS, 1, KIN, kChemSharedMat>(A, cnt);
    else if (cnt <= kChemShortList)
        chem_list_groups<NS, 8, KIN>(A, cnt);
    else
        chem_list_groups<NS, 4, KIN>(A, cnt);
}

// Chemistry of every fluid cell for LBMGPU_CHEM_ROSENBROCK handles, one thread per cell,
// beside the transport part of the collision parameters (k_mc_props<CHEM_OFF>), from the
// state the collision forms from the record (mc_chem_state):
//   SUR = false: the stiff integrator (ROS2) itself;
//   SUR = true : the surrogate's prediction where the gate passes it (element projection,
//                output gate), the cells it does not cover and the audited ones appended
//                to the integrator list for k_mc_chem_list.
// A kernel of its own, so that its time (with the surrogate's kernels) is the chemistry's
// share of the step, and the transport kernel keeps its own occupancy.
// One thread per cell.  The integrator's vectors are sized by the species count at compile
// time (ros2_advance_k) so that they stay in registers, two blocks per SM.  KIN: the compiled
// kinetics of the handle's mechanism (gen_kinetics.py), void for the tables; with it the
// iteration matrix of each thread lives in shared memory (kChemSharedMat), otherwise in the
// thread's local memory.
// The surrogate's instance (SUR: no integrator in it) holds far less per thread and runs four
// blocks per SM.
// PRED false: launched only while the surrogate's predictions are not in use (mode != 1).
template <int NS, bool SUR, class KIN = void, bool PRED = true>
__global__ void __launch_bounds__(kBlock, SUR ? 4 : 2) k_mc_chem(McArgs A) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= A.ncell || !(A.cflag[n] & CF_FLUID)) return;
    double rho, rho_a[NS], Y[NS], T_si, rho_si, P_si;
    mc_chem_state<NS>(A, n, rho, rho_a, Y, T_si, rho_si, P_si);
    constexpr bool smat = kChemSharedMat && !std::is_void_v<KIN>;
    mc_chem_ros2<NS, McArgs, !SUR, 1, KIN, smat, PRED>(A, n, rho, rho_a, Y, T_si, rho_si, P_si, SUR);
}

// The reference's explicit chemistry of every fluid cell (mc_chem_explicit), one thread per cell.
// NET: the net production rates -- the compiled kinetics of the handle's mechanism, or the dense
// tables (gas::DenseNet).  A kernel of its own: inside the transport kernel the table-driven rates
// (a RateT per temperature, 2.4 kB of local arrays) took 135 of 202 us at 512 cells and 180 of 248 us
// at 33 k cells; here transport and chemistry together take 79 and 126 us.
template <int NS, typename S, class NET>
__global__ void __launch_bounds__(kBlock, 2) k_mc_explicit(McArgsT<S, double> A) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= A.ncell || !(A.cflag[n] & CF_FLUID)) return;
    if constexpr (std::is_same_v<NET, gas::DenseNet<NS>>)
        mc_chem_explicit<NS>(A, n, NET{*A.tab});
    else
        mc_chem_explicit<NS>(A, n, NET{});
}

// The stiff chemistry over the compiled kinetics of the handle's mechanism, where the library
// has them for it (kinetics_h2_air_9.cuh): every cell (k_mc_chem) or the integrator list
// (k_mc_chem_list).  Returns false when the handle's mechanism is not compiled.
template <int NS>
bool launch_compiled_chem(lbmgpu *h, const McArgs &A, unsigned grid, bool list, cudaStream_t st) {
    if constexpr (NS == kin_h2_air_9::NS) {
        using KinH2 = kin_h2_air_9::Kinetics;
        if (h->kin != KIN_H2_AIR_9) return false;
        constexpr size_t sm = chem_smem_bytes<NS, KinH2>();
        // the launches below report a refused attribute as a launch error
        if (list) {
            if (sm > 48 * 1024)
                (void)cudaFuncSetAttribute(k_mc_chem_list<NS, KinH2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sm);
            k_mc_chem_list<NS, KinH2><<<grid, kBlock, sm, st>>>(A);
        } else if (A.sur.mode == 1) {
            if (sm > 48 * 1024)
                (void)cudaFuncSetAttribute(k_mc_chem<NS, false, KinH2>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            k_mc_chem<NS, false, KinH2><<<grid, kBlock, sm, st>>>(A);
        } else {
            if (sm > 48 * 1024)
                (void)cudaFuncSetAttribute(k_mc_chem<NS, false, KinH2, false>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            k_mc_chem<NS, false, KinH2, false><<<grid, kBlock, sm, st>>>(A);
        }
        return true;
    }
    return false;
}

}  // namespace

namespace lbmh {

template <int NS>
int chem_step(lbmgpu *h, const lbm::McArgs &A, cudaStream_t st) {
    const unsigned gp = grid_for(h->g.ncell);
    EvPair ec{};
    ev_begin(h, K_CHEM, ec, st);
    if (A.sur.mode == 1 && A.sur.ilist)
        k_mc_chem<NS, true><<<gp, kBlock, 0, st>>>(A);
    else if (!launch_compiled_chem<NS>(h, A, gp, false, st))
        k_mc_chem<NS, false><<<gp, kBlock, 0, st>>>(A);
    ev_end(h, ec, st);
    CK(cudaGetLastError());
    if (A.sur.ilist) {
        EvPair ei{};
        ev_begin(h, K_SURROGATE, ei, st);
        if (!launch_compiled_chem<NS>(h, A, 148 * 8, true, st))
            k_mc_chem_list<NS><<<148 * 8, kBlock, 0, st>>>(A);
        ev_end(h, ei, st);
        CK(cudaGetLastError());
    }
    return 0;
}

template <int NS, typename S>
int explicit_step(lbmgpu *h, const lbm::McArgsT<S, double> &A, cudaStream_t st) {
    const unsigned gp = grid_for(h->g.ncell);
    EvPair ec{};
    ev_begin(h, K_CHEM, ec, st);
    bool compiled = false;
    if constexpr (NS == kin_h2_air_9::NS) {
        if (h->kin == KIN_H2_AIR_9) {
            k_mc_explicit<NS, S, kin_h2_air_9::Kinetics><<<gp, kBlock, 0, st>>>(A);
            compiled = true;
        }
    }
    if (!compiled) k_mc_explicit<NS, S, gas::DenseNet<NS>><<<gp, kBlock, 0, st>>>(A);
    ev_end(h, ec, st);
    CK(cudaGetLastError());
    return 0;
}

}  // namespace lbmh
