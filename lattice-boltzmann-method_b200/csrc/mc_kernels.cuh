// lbmgpu, multicomponent path: the device kernels around the per-cell functions of
// mc_cell.cuh and their launches, for one species count NS (McOps<NS>, instantiated in
// mc_ns<NS>.cu; the handle operations that dispatch to them are in mc.cu).
//
// Reference path replaced (farrasarira/Lattice-Boltzmann-Method, MULTICOMP on):
//   LBM::Collide_Species + LBM::Collide   src/lbm-collision.cpp:191-526 -> k_mc_props, the stiff
//                                          chemistry (mc_chem.cuh), k_mc_eflux, k_mc_relax
//   LBM::Streaming + LBM::calculate_moment src/lbm-streaming.cpp, src/lbm-moment.cpp:193-377
//                                          -> k_mc_gather (pull + population sums),
//                                             k_mc_diffuse and k_mc_thermo (mc_moments.cuh)
//   LBM::Init                              src/lbm-init.cpp:85-146 -> k_mc_init
//   LBM::Streaming + LBM::TMS_BC + LBM::calculate_moment of the cells with a boundary
//   upstream (src/lbm-bc.cpp:122-1110, src/impose_nscbc.cpp) -> k_mc_special (mc_special.cuh)
#pragma once
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "halo.cuh"
#include "handle.cuh"
#include "mc_bc.cuh"
#include "mc_cell.cuh"
#include "launch.cuh"
#include "mc_eflux.cuh"
#include "mc_moments.cuh"
#include "mc_ops.cuh"
#include "mc_relax.cuh"
#include "surrogate_host.cuh"

namespace {

using namespace lbm;
using namespace lbmh;

// Transport part of the collision parameters of every fluid cell (the chemistry runs in kernels of
// its own, mc_chem.cuh), one thread per cell.  Bound by the latency of its FP64 chains and of the record
// loads, not by HBM; three blocks per SM (168 registers), the species loops unrolled, so that no
// per-species array is indexed in local memory (nine species, FP64: 184 B of spills; FP32: 8 B), the
// species velocities loaded where the Maxwell-Stefan force uses them.  FP64 storage, 48 x 40 x 37 cells:
// 189 us with rolled loops (920 B of local arrays) and 400 divisions per cell, 119 us unrolled, 110 us
// with the diffusion coefficients' pairs rolled again (mc_transport_f64); FP32 storage, 96^3: 523 -> 502 us.
template <int NS, typename S>
__global__ void __launch_bounds__(kBlock, 3) k_mc_props(McArgsT<S, double> A) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    lbmh::step_begin();
    if (n >= A.ncell || !(A.cflag[n] & CF_FLUID)) return;
    mc_props_cell<NS, CHEM_OFF, false>(A, n);
}

template <int NS, typename S>
__global__ void __launch_bounds__(kBlock) k_mc_init(McArgsT<S, double> A, double *rec0, double *rec1, S *pop0) {
    const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= A.ncell) return;
    mc_init_cell<NS>(A, n, rec0, rec1, pop0);
}


__device__ __forceinline__ double ldd(const char *rec, long off) { return *reinterpret_cast<const double *>(rec + off); }
__device__ __forceinline__ void std_(char *rec, long off, double v) { *reinterpret_cast<double *>(rec + off) = v; }

// Staging layout of a chunk of cnt cells: cnt mixture records, then cnt records of each
// species in turn.
template <int NS, typename S>
__global__ void k_mc_unpack(McArgsT<S, double> A, MixOff mo, SpOff so, const char *__restrict__ stage, long n0, long n1,
                            double *rec0, double *rec1, S *pop0, S *pop1) {
    const long n = n0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n1) return;
    const long cnt = n1 - n0;
    const char *mr = stage + (n - n0) * mo.size;
    auto pr = [&](int plane, double v) {
        put(A, rec0, plane, n, v);
        put(A, rec1, plane, n, v);
    };
    const double rho = ldd(mr, mo.rho), T = ldd(mr, mo.temp);
    const double um[3] = {ldd(mr, mo.u), ldd(mr, mo.v), ldd(mr, mo.w)};
    pr(RM_RHO, rho);
    pr(RM_U, um[0]);
    pr(RM_V, um[1]);
    pr(RM_W, um[2]);
    pr(RM_T, T);
    pr(RM_P, ldd(mr, mo.p));
    pr(RM_RHOE, ldd(mr, mo.rhoe));
    const int pi[6][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}};
    for (int q = 0; q < 6; ++q) pr(RM_P00 + q, ldd(mr, mo.p_tensor + 8 * (3 * pi[q][0] + pi[q][1])));
    pr(RM_HRR, ldd(mr, mo.HRR));
    const bool fluid = A.type[n] == T_F;  // the cell classification follows the whole upload
    double rho_a[NS], ua[NS][3];
    for (int a = 0; a < NS; ++a) {
        const char *sr = stage + cnt * mo.size + ((long)a * cnt + (n - n0)) * so.size;
        rho_a[a] = ldd(sr, so.rho);
        ua[a][0] = ldd(sr, so.u);
        ua[a][1] = ldd(sr, so.v);
        ua[a][2] = ldd(sr, so.w);
        pr(rs(a, RS_RHO), rho_a[a]);
        for (int d = 0; d < 3; ++d) pr(rs(a, RS_UX + d), ua[a][d]);
        pr(rs(a, RS_X), ldd(sr, so.X));
        if (fluid)
            for (int l = 0; l < 27; ++l) {
                stpop(A, pop0, 27 * a + l, n, ldd(sr, so.f + 8 * l));
                stpop(A, pop1, 27 * a + l, n, ldd(sr, so.fpc + 8 * l));
            }
    }
    store_face_terms<NS>(A, rec0, n, A.type[n], rho, um, T, rho_a, ua);
    store_face_terms<NS>(A, rec1, n, A.type[n], rho, um, T, rho_a, ua);
    if (fluid)
        for (int l = 0; l < 27; ++l) {
            stpop(A, pop0, 27 * NS + l, n, ldd(mr, mo.g + 8 * l));
            stpop(A, pop1, 27 * NS + l, n, ldd(mr, mo.gpc + 8 * l));
        }
}

// pop_now: what the cell's populations are taken from (pulled when `stepped`, in place
// otherwise); pop_pc: the post-collision populations (fpc, gpc).
template <int NS, typename S>
__global__ void k_mc_pack(McArgsT<S, double> A, MixOff mo, SpOff so, char *__restrict__ stage, long n0, long n1,
                          const double *rec, const S *pop_now, const S *pop_pc, const S *bst, int stepped) {
    const long n = n0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n1) return;
    const long cnt = n1 - n0;
    char *mr = stage + (n - n0) * mo.size;
    auto get = [&](int plane) { return (double)rec[(long)plane * A.ncell + n]; };
    std_(mr, mo.rho, get(RM_RHO));
    std_(mr, mo.u, get(RM_U));
    std_(mr, mo.v, get(RM_V));
    std_(mr, mo.w, get(RM_W));
    std_(mr, mo.temp, get(RM_T));
    std_(mr, mo.p, get(RM_P));
    std_(mr, mo.rhoe, get(RM_RHOE));
    std_(mr, mo.HRR, get(RM_HRR));
    const int full[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    for (int q = 0; q < 9; ++q) std_(mr, mo.p_tensor + 8 * q, get(RM_P00 + full[q]));
    const bool fluid = A.cflag[n] & CF_FLUID;
    const bool special = stepped && (A.cflag[n] & CF_SPECIAL);
    const long bs = special ? (long)A.bid[n] : 0;
    McPull pp;
    mc_pull(A, n, pp);
    // the cell's populations: kept in the special-cell store, pulled, or in place
    auto now = [&](int plane, int l) {
        if (special) return ldpop_b(A, bst, plane, bs);
        return ldpop(A, pop_now, plane, stepped ? pull_idx(pp, l) : n);
    };
    for (int a = 0; a < NS; ++a) {
        char *sr = stage + cnt * mo.size + ((long)a * cnt + (n - n0)) * so.size;
        std_(sr, so.rho, get(rs(a, RS_RHO)));
        std_(sr, so.u, get(rs(a, RS_UX)));
        std_(sr, so.v, get(rs(a, RS_UX + 1)));
        std_(sr, so.w, get(rs(a, RS_UX + 2)));
        std_(sr, so.X, get(rs(a, RS_X)));
        if (!fluid) continue;
        for (int l = 0; l < 27; ++l) {
            const int plane = 27 * a + l;
            std_(sr, so.f + 8 * l, now(plane, l));
            std_(sr, so.fpc + 8 * l, ldpop(A, pop_pc, plane, n));
        }
    }
    if (!fluid) return;
    double q3[3] = {0, 0, 0};
    for (int l = 0; l < 27; ++l) {
        const int plane = 27 * NS + l;
        const double gv = now(plane, l);
        std_(mr, mo.g + 8 * l, gv);
        std_(mr, mo.gpc + 8 * l, ldpop(A, pop_pc, plane, n));
        q3[0] += gv * cx(l);
        q3[1] += gv * cy(l);
        q3[2] += gv * cz(l);
    }
    for (int q = 0; q < 3; ++q) std_(mr, mo.energy_flux + 8 * q, q3[q]);
}

// The records of cells [c0, c1) -- the caller's arrays start at cell c0 -- into the device
// state, one staging chunk at a time.
template <int NS, typename S>
int upload_t(lbmgpu *h, const char *hm, const void *const *species, long c0, long c1) {
    const size_t ms = h->mo.size, ss = h->so.size;
    McArgsT<S, double> A = base_args<S>(h);
    // pageable caller memory goes through the pinned bounce buffer, filled by host threads
    // (a copy from pageable memory would otherwise be staged by the driver, one thread);
    // page-locked caller memory is copied directly
    bool pinned = host_pinned(hm);
    for (int a = 0; a < h->ns; ++a) pinned = pinned && host_pinned(species[a]);
    // host threads fill one bounce buffer while the other's copy is under way; fork and join mark the two
    // buffers' copies (no step is running during an upload)
    const long step = pinned ? (long)h->stage_cells : transfer_chunk(h, c1 - c0);
    const cudaEvent_t copied[2] = {h->fork, h->join};
    if (!pinned) CK(cudaStreamSynchronize(h->stream));  // the bounce buffers' earlier copies have gone
    long chunk = 0;
    for (long n0 = c0; n0 < c1; n0 += step, ++chunk) {
        const long n1 = std::min<long>(c1, n0 + step), cnt = n1 - n0;
        char *const bounce = chunk & 1 ? h->bounce2 : h->bounce;
        if (pinned) {
            CK(cudaMemcpyAsync(h->stage, hm + (n0 - c0) * ms, cnt * ms, cudaMemcpyHostToDevice, h->stream));
            for (int a = 0; a < h->ns; ++a)
                CK(cudaMemcpyAsync(h->stage + cnt * ms + (size_t)a * cnt * ss,
                                   static_cast<const char *>(species[a]) + (n0 - c0) * ss, cnt * ss,
                                   cudaMemcpyHostToDevice, h->stream));
        } else {
            if (chunk >= 2) CK(cudaEventSynchronize(copied[chunk & 1]));  // the buffer's previous chunk has gone
            const long nb = (long)h->ns + 1;  // the mixture block, then each species' block
            host_parallel_for(nb * 64, [&](long lo, long hi) {
                for (long q = lo; q < hi; ++q) {
                    const long blk = q / 64, part = q % 64;
                    const size_t sz = blk == 0 ? ms : ss;
                    const char *src = blk == 0 ? hm : static_cast<const char *>(species[blk - 1]);
                    char *dst = bounce + (blk == 0 ? 0 : cnt * ms + (size_t)(blk - 1) * cnt * ss);
                    const long r0 = cnt * part / 64, r1 = cnt * (part + 1) / 64;
                    std::memcpy(dst + r0 * sz, src + (n0 - c0 + r0) * sz, (r1 - r0) * sz);
                }
            }, 1);
            CK(cudaMemcpyAsync(h->stage, bounce, cnt * (ms + (size_t)h->ns * ss), cudaMemcpyHostToDevice, h->stream));
            CK(cudaEventRecord(copied[chunk & 1], h->stream));
        }
        EvPair ep{};
        ev_begin(h, K_OTHER, ep);
        k_mc_unpack<NS, S><<<grid_for(cnt), kBlock, 0, h->stream>>>(A, h->mo, h->so, h->stage, n0, n1, h->mom[0],
                                                                     h->mom[1], popb<S>(h, 0), popb<S>(h, 1));
        ev_end(h, ep);
        CK(cudaGetLastError());
    }
    return 0;
}

template <int NS, typename S>
int pack_chunk(lbmgpu *h, long n0, long n1, bool stepped) {
    McArgsT<S, double> A = base_args<S>(h);
    const int c = h->cur;
    const S *pc = stepped ? popb<S>(h, c) : popb<S>(h, 1 - c);
    // the records' padding bytes come out as zeros, not as what the staging held before
    CK(cudaMemsetAsync(h->stage, 0, (size_t)(n1 - n0) * (h->mo.size + (size_t)h->ns * h->so.size), h->stream));
    EvPair ep{};
    ev_begin(h, K_OTHER, ep);
    k_mc_pack<NS, S><<<grid_for(n1 - n0), kBlock, 0, h->stream>>>(A, h->mo, h->so, h->stage, n0, n1, h->mom[c],
                                                                   popb<S>(h, c), pc, bstb<S>(h, c), stepped ? 1 : 0);
    ev_end(h, ep);
    CK(cudaGetLastError());
    return 0;
}

template <int NS, typename S>
int init_t(lbmgpu *h) {
    McArgsT<S, double> A = base_args<S>(h);
    const int c = h->cur;
    EvPair ep{};
    ev_begin(h, K_OTHER, ep);
    k_mc_init<NS, S><<<grid_for(h->g.ncell), kBlock, 0, h->stream>>>(A, h->mom[c], h->mom[1 - c],
                                                                      popb<S>(h, c));
    ev_end(h, ep);
    CK(cudaGetLastError());
    return 0;
}

template <int NS, typename S>
int collide_t(lbmgpu *h) {
    const int c = h->cur, x = 1 - c;
    McArgsT<S, double> A = base_args<S>(h);
    const bool local = h->pack_mode != PK_STEPPED;
    A.pop_src = popb<S>(h, c);
    A.pop_dst = popb<S>(h, x);
    A.pop_prev = local ? nullptr : popb<S>(h, c);
    A.rec_cur = h->mom[c];
    A.rec_nxt = h->mom[x];
    A.local = local ? 1 : 0;
    A.bst_cur = bstb<S>(h, c);
    const int rs_ = sur_prepare_t<S>(h, A);
    if (rs_) return rs_;
    const unsigned gp = grid_for(h->g.ncell);
    // The chemistry runs on the side stream beside the transport and energy-flux kernels: they read the
    // same record and write different parameters, and on small lattices neither fills the device
    // (8^3, explicit chemistry: 137 -> 97 us a step).  While kernels are timed they run in turn.
    const bool beside = h->chem != CHEM_OFF && !h->prof;
    if (beside) {
        CK(cudaEventRecord(h->fork, h->stream));
        CK(cudaStreamWaitEvent(h->side, h->fork, 0));
    }
    const cudaStream_t cs = beside ? h->side : h->stream;
    if (h->chem == CHEM_REF_EXPLICIT) {
        const int rc_ = explicit_step<NS, S>(h, A, cs);
        if (rc_) return rc_;
    } else if (h->chem == CHEM_ROSENBROCK) {
        McArgsT<double, double> C = base_args<double>(h);  // no populations in it: one instance for both storages
        C.rec_cur = A.rec_cur;
        C.rec_nxt = A.rec_nxt;
        C.sur = A.sur;
        const int rc_ = chem_step<NS>(h, C, cs);
        if (rc_) return rc_;
    }
    if (beside) CK(cudaEventRecord(h->join, h->side));
    EvPair ep{};
    ev_begin(h, K_PROPS, ep);
    // after the last step's moments, if nothing was put on the stream between
    CK(launch_next(!h->prof && !beside && h->nb == 0 && !local, k_mc_props<NS, S>, gp, kBlock, 0, h->stream, A));
    ev_end(h, ep);
    EvPair ee{};
    ev_begin(h, K_EFLUX, ee);
    CK(launch_next(!h->prof, k_mc_eflux<NS, S>, gp, kBlock, 0, h->stream, A));
    ev_end(h, ee);
    if (beside) CK(cudaStreamWaitEvent(h->stream, h->join, 0));
    EvPair er{};
    ev_begin(h, K_COLLIDE, er);
    CK(launch_next(!h->prof && !beside, h->chem == CHEM_OFF ? k_mc_relax<NS, false, S> : k_mc_relax<NS, true, S>,
                   dim3(gp, NS + 1), kBlock, 0, h->stream, A));
    ev_end(h, er);
    return 0;
}

template <int NS, typename S>
int stream_t(lbmgpu *h) {
    const int c = h->cur, x = 1 - c;
    McArgsT<S, double> A = base_args<S>(h);
    A.pop_src = popb<S>(h, x);
    A.rec_cur = h->mom[c];
    A.rec_nxt = h->mom[x];
    // The boundary cells run on the side stream beside the interior's gather and solve:
    // the two sets of cells are disjoint, and both read only the post-collision populations
    // and the previous records, so the latency-bound boundary kernel overlaps them; the
    // handle's stream waits for it before anything that follows.
    if (h->nb > 0) {
        McArgsT<S, double> B = A;
        B.bst_cur = bstb<S>(h, c);
        B.bst_nxt = bstb<S>(h, x);
        CK(cudaEventRecord(h->fork, h->stream));
        CK(cudaStreamWaitEvent(h->side, h->fork, 0));
        const int rb = special_step<NS, S>(h, B);
        if (rb) return rb;
        CK(cudaEventRecord(h->join, h->side));
    }
    EvPair ep{};
    ev_begin(h, K_STREAM_MOMENT, ep);
    CK(launch_next(!h->prof && h->nb == 0, k_mc_gather<NS, S>, (unsigned)((h->g.ncell + kGatherCells - 1) / kGatherCells),
                   kGatherCells * (NS + 1), 0, h->stream, A));
    ev_end(h, ep);
    EvPair es{};
    ev_begin(h, K_SOLVE, es);
    CK(launch_next(!h->prof, k_mc_diffuse<NS, S>, grid_for(h->g.ncell), kBlock, 0, h->stream, A));
    ev_end(h, es);
    EvPair et{};
    ev_begin(h, K_SOLVE, et);
    CK(launch_next(!h->prof, k_mc_thermo<NS, S>, grid_for(h->g.ncell), kBlock, 0, h->stream, A));
    ev_end(h, et);
    if (h->nb > 0) CK(cudaStreamWaitEvent(h->stream, h->join, 0));
    return 0;
}

// Slab faces (halo.cuh): one thread per cell of the face plane.
template <int NS, typename S>
__global__ void k_halo_pack(McArgsT<S, double> A, const S *pop, const double *rec, int face, int what,
                            double *__restrict__ buf) {
    const long jk = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (jk >= (long)A.Ny * A.Nz) return;
    halo_pack_cell<NS>(A, pop, rec, face, what, jk, buf);
}
template <int NS, typename S>
__global__ void k_halo_unpack(McArgsT<S, double> A, S *pop, double *rec, int face, int what,
                              const double *__restrict__ buf) {
    const long jk = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (jk >= (long)A.Ny * A.Nz) return;
    halo_unpack_cell<NS>(A, pop, rec, face, what, jk, buf);
}

// populations: the post-collision buffer the coming stream reads (between Collide and
// calculate_moment); record: the current step's record (between steps)
template <int NS, typename S>
int halo_t(lbmgpu *h, int face, int what, double *buf, bool pack) {
    McArgsT<S, double> A = base_args<S>(h);
    S *pop = popb<S>(h, 1 - h->cur);
    double *rec = h->mom[h->cur];
    const long plane = (long)h->g.Ny * h->g.Nz;
    EvPair ep{};
    ev_begin(h, K_OTHER, ep);
    if (pack)
        k_halo_pack<NS, S><<<grid_for(plane), kBlock, 0, h->stream>>>(A, pop, rec, face, what, buf);
    else
        k_halo_unpack<NS, S><<<grid_for(plane), kBlock, 0, h->stream>>>(A, pop, rec, face, what, buf);
    ev_end(h, ep);
    CK(cudaGetLastError());
    return 0;
}

}  // namespace

namespace lbmh {

template <int NS>
int McOps<NS>::upload(lbmgpu *h, const char *hm, const void *const *species, long c0, long c1) {
    return h->fp32 ? upload_t<NS, float>(h, hm, species, c0, c1) : upload_t<NS, double>(h, hm, species, c0, c1);
}
template <int NS>
int McOps<NS>::pack(lbmgpu *h, long n0, long n1, bool stepped) {
    return h->fp32 ? pack_chunk<NS, float>(h, n0, n1, stepped) : pack_chunk<NS, double>(h, n0, n1, stepped);
}
template <int NS>
int McOps<NS>::init(lbmgpu *h) {
    return h->fp32 ? init_t<NS, float>(h) : init_t<NS, double>(h);
}
template <int NS>
int McOps<NS>::collide(lbmgpu *h) {
    return h->fp32 ? collide_t<NS, float>(h) : collide_t<NS, double>(h);
}
template <int NS>
int McOps<NS>::stream(lbmgpu *h) {
    return h->fp32 ? stream_t<NS, float>(h) : stream_t<NS, double>(h);
}
template <int NS>
int McOps<NS>::halo(lbmgpu *h, int face, int what, double *buf, bool pack) {
    return h->fp32 ? halo_t<NS, float>(h, face, what, buf, pack) : halo_t<NS, double>(h, face, what, buf, pack);
}

}  // namespace lbmh
