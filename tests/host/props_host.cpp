// Host build of the collision parameters' two FP64 forms (csrc/mc_cell.cuh, mc_transport_f64), for
// tests/test_transport_forms.py.
#include "mc_cell.cuh"

namespace {
template <int NS>
int run(const lbmgpu_mech *m, float dx, float dt, long n, const double *rec, int exact, double *props) {
    using namespace lbm;
    gas::Tables tab{};
    gas::make_tables(*m, tab);
    McArgs A{};
    A.U = units_from_dx_dt(dx, dt);
    set_lattice_constants(tab, A.U);
    A.ncell = n;
    A.ns = NS;
    A.dt = 1;
    A.tab = &tab;
    A.rec_cur = rec;
    A.props = props;
    for (long c = 0; c < n; ++c)
        if (exact)
            mc_props_cell<NS, CHEM_OFF, true>(A, c);
        else
            mc_props_cell<NS, CHEM_OFF, false>(A, c);
    return pr_count<NS>();
}
}  // namespace

extern "C" int collision_params(const lbmgpu_mech *m, float dx, float dt, long n, const double *rec, int exact, double *props) {
    return m->n_species == 9 ? run<9>(m, dx, dt, n, rec, exact, props) : run<6>(m, dx, dt, n, rec, exact, props);
}
